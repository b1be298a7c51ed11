"""The work that users of this framework have it do, as timed cases.

A case names one public entry point and its sizes.  Synthetic data comes from
``glphase_gb300.synth_device`` (Li-Stephens mosaics, Poisson depth, binomial
reads), whose distributions are those of the repository's benchmark.  A pass
of a generation is what the phasing loop does between two readings of its
state: one generation, the haplotype swap, the wait that collects errors.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from glphase_gb300 import batch as gbatch
from glphase_gb300 import glpack, hmmlike, model, phase, synth, synth_device

# ---------------------------------------------------------------------------
# cases


def listed():
    return [
        # the simple-GL run of three samples and three sites: launches and latency only
        {"name": "tiny_generation", "kind": "generation", "N": 3, "S": 3, "panel": 0, "C": 100,
         "knn": 0, "vq": False, "pen": 1.0, "depth": 4.0, "founders": 40},
        # one window of a small cohort, surrogates from all other samples
        {"name": "plain_generation", "kind": "generation", "N": 256, "S": 1024, "panel": 0,
         "C": 100, "knn": 0, "vq": False, "pen": 1.0, "depth": 4.0, "founders": 40},
        # a large low-coverage cohort, surrogates from the K nearest haplotypes
        {"name": "batched_generation", "kind": "generation", "N": 10000, "S": 4096, "panel": 0,
         "C": 100, "knn": 200, "vq": False, "pen": 1.0, "depth": 2.0, "founders": 80},
        # burn-in generation (annealed penalty) on 4-bit GL codes, sites not a whole number of words
        {"name": "vq_burnin_generation", "kind": "generation", "N": 3001, "S": 4000, "panel": 0,
         "C": 100, "knn": 200, "vq": True, "pen": 0.140625, "depth": 2.0, "founders": 80},
        # samples phased against a reference panel
        {"name": "panel_generation", "kind": "generation", "N": 2000, "S": 8192, "panel": 10000,
         "C": 100, "knn": 0, "vq": False, "pen": 1.0, "depth": 4.0, "founders": 80},
        # chunks of uneven size in one prepared launch (serving, many windows)
        {"name": "uneven_batch", "kind": "batch", "chunks": 8, "N_lo": 100, "N_hi": 2000,
         "S_lo": 512, "S_hi": 8192, "C": 100},
        # the reference's device call: host buffers, 4-bit GL codes, its 1,024-site window
        {"name": "dropin_call", "kind": "dropin", "N": 500, "S": 1024, "C": 100},
        # the neighbour table of the large cohort, Hamming distance
        {"name": "knn_hamming", "kind": "knn", "H": 20000, "S": 4096, "K": 200,
         "metric": "hamming"},
        # the neighbour table of 2,495 samples by shared tract length (-T)
        {"name": "knn_tract", "kind": "knn", "H": 4990, "S": 1024, "K": 200, "metric": "tract"},
        # allele tallies of the sampling generations and the final probabilities
        {"name": "tally_result", "kind": "tally", "N": 10000, "S": 4096, "samples": 4},
        # codebook training and packing of a cohort's GLs
        {"name": "vq_codec", "kind": "codec", "N": 2000, "S": 8192},
        # a whole phasing run of a small cohort, host arrays in and out
        {"name": "phase_run", "kind": "phase", "N": 60, "S": 1000, "panel": 0, "C": 100,
         "B": 5, "I": 5, "M": 20, "knn": 0, "recluster": 0, "metric": "hamming"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["generation"] * 6 + ["batch", "dropin", "knn", "knn", "tally", "codec",
                                            "phase"])
    if kind == "generation":
        S = _log(rng, 3, 12288)
        N = _log(rng, 3, max(4, min(10000, 30_000_000 // S)))
        knn = rng.choice([0, _log(rng, 20, 200)])
        panel = rng.choice([0, 2 * _log(rng, 50, 5000)])
        knn = min(knn, 2 * ((2 * N + panel - 2) // 2 // 2))
        return {"kind": kind, "N": N, "S": S, "panel": panel,
                "C": rng.choice([20, 50, 100, 100]), "knn": knn,
                "vq": rng.random() < 0.25, "pen": rng.choice([1.0, 1.0, 0.140625, 0.5625]),
                "depth": rng.choice([2.0, 4.0, 8.0]), "founders": rng.randrange(20, 81)}
    if kind == "batch":
        S_hi = 64 * _log(rng, 9, 192)
        return {"kind": kind, "chunks": rng.randrange(2, 9), "N_lo": 100,
                "N_hi": _log(rng, 150, max(160, min(2000, 16_000_000 // S_hi))), "S_lo": 512,
                "S_hi": S_hi, "C": 100}
    if kind == "dropin":
        return {"kind": kind, "N": _log(rng, 3, 2000), "S": _log(rng, 8, 1024),
                "C": rng.choice([50, 100])}
    if kind == "knn":
        H = 2 * _log(rng, 30, 7000)
        return {"kind": kind, "H": H, "S": _log(rng, 64, 4096),
                "K": min(_log(rng, 10, 200), H - 2 - H % 2),
                "metric": rng.choice(["hamming", "tract"])}
    if kind == "tally":
        N = _log(rng, 60, 8000)
        return {"kind": kind, "N": N, "S": _log(rng, 100, min(16384, 32_000_000 // N)),
                "samples": rng.randrange(1, 6)}
    if kind == "codec":
        N = _log(rng, 60, 4000)
        return {"kind": kind, "N": N, "S": _log(rng, 100, min(16384, 16_000_000 // N))}
    N = _log(rng, 10, 200)
    knn = rng.choice([0, min(20, 2 * (N // 2))])
    return {"kind": "phase", "N": N, "S": _log(rng, 64, 1500), "panel": rng.choice([0, 120]),
            "C": rng.choice([50, 100]), "B": 5, "I": rng.randrange(0, 6),
            "M": rng.randrange(5, 21), "knn": knn, "recluster": rng.choice([0, 4]) if knn else 0,
            "metric": rng.choice(["hamming", "tract"])}


# ---------------------------------------------------------------------------
# inputs


def _workload(case):
    return synth.Workload("case", N=case["N"], S=case["S"], founders=case.get("founders", 60),
                          depth=case.get("depth", 4.0), burnin=8, sampling=16,
                          panel_haps=case.get("panel", 0))


def _chunk(case, seed):
    return synth_device.generate(_workload(case), case["N"], case["S"], seed)


def _panel_bits(H, S, seed, flips=0.1):
    """Haplotypes as the sampler holds them: mosaics of founders with the
    errors that low-coverage GLs leave in them.  [H][S] uint8 on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    F = 80
    freq = torch.from_numpy(np.random.default_rng(seed).beta(0.5, 0.5, size=S)).cuda()
    founders = torch.rand((F, S), generator=g, device="cuda") < freq[None, :]
    switch = torch.rand((H, S), generator=g, device="cuda") < 1e-3
    switch[:, 0] = True
    col = torch.arange(S, device="cuda")
    at = torch.where(switch, col[None, :], torch.zeros_like(col)[None, :]).cummax(dim=1).values
    src = torch.randint(0, F, (H, S), generator=g, device="cuda").gather(1, at)
    bits = founders[src, col[None, :]]
    noise = torch.rand((H, S), generator=g, device="cuda") < flips
    other = torch.rand((H, S), generator=g, device="cuda") < freq[None, :]
    return torch.where(noise, other, bits).to(torch.uint8)


def _packed(bits):
    return synth_device.pack_bits_device(bits)


def _host_words(t):
    return t.cpu().numpy().view(np.uint64)


def _gl_codes(dev, prob, seed):
    """4-bit codes and the codebook of the GLs, as a VQ run packs them once."""
    vq = glpack.GLVQ(prob.reshape(-1, 3), np.random.default_rng(seed), device=dev)
    N, S = prob.shape[0], prob.shape[1]
    out = torch.zeros(((S + 7) // 8, N), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    dev._c(dev.L.glp_vq_pack(dev.ctx, prob.data_ptr(), N, S, vq.codebook.ctypes.data, 16, 4,
                             out.data_ptr()))
    dev._c(dev.L.glp_finish(dev.ctx))
    return out.cpu().numpy().view(np.uint32), vq.codebook


def _batch_shapes(case, seed):
    rng = np.random.default_rng(seed)
    n = case["chunks"]
    S = 64 * rng.integers(case["S_lo"] // 64, case["S_hi"] // 64 + 1, size=n)
    N = rng.integers(case["N_lo"], case["N_hi"] + 1, size=n)
    # the same amount of work for every seed: the middle of both ranges last
    S[-1], N[-1] = case["S_hi"], case["N_hi"]
    return [(int(a), int(b)) for a, b in zip(N, S)]


def _prepare_generation(case, seed):
    ch = _chunk(case, seed)
    packed = codebook = None
    if case["vq"]:
        dev = hmmlike.HMMLikeCUDA(0)
        packed, codebook = _gl_codes(dev, ch.prob, seed)
        dev.cleanup()
    eng = hmmlike.Engine(ch.emit.cpu().numpy(), ch.prob.cpu().numpy(), ch.tran, ch.pc,
                         _host_words(ch.haps), case["C"], packed=packed, codebook=codebook)
    nbr = eng.knn(case["knn"]) if case["knn"] else None
    eng.finish()
    return {"eng": eng, "nbr": nbr, "g": 0, "seed": int(seed)}


class _Batch(gbatch.PreparedBatch):
    """A prepared batch that gives its device memory back with itself."""

    def __del__(self):
        self.close()
        for p in self.problems:
            p.close()


def _prepare_batch(case, seed):
    dev = hmmlike.HMMLikeCUDA(0)
    problems = []
    for i, (N, S) in enumerate(_batch_shapes(case, 4)):
        ch = synth_device.generate(synth.Workload("chunk", N=N, S=S, founders=40, depth=4.0,
                                                  burnin=8, sampling=24), N, S, 100 * seed + i)
        problems.append(gbatch.DeviceProblem(dev, ch, case["C"], seed=1000 * seed + i, burnin=8))
    torch.cuda.synchronize()
    return {"dev": dev, "problems": problems, "batch": _Batch(dev, problems, 8)}


def _prepare_dropin(case, seed):
    N, S, C = case["N"], case["S"], case["C"]
    ch = _chunk(case, seed)
    dev = hmmlike.HMMLikeCUDA(0)
    packed, codebook = _gl_codes(dev, ch.prob, seed)
    dev.copy_tran_to_device(ch.tran)
    dev.copy_mutation_mat_to_device(ch.pc)
    dev.copy_code_book_to_device(codebook)
    dev.copy_packed_gls_to_device(packed)
    quad, props = synth.uniform_proposals(N, ch.H, C, np.random.default_rng(seed))
    return {"dev": dev, "panel": _host_words(ch.haps), "quad": quad, "props": props,
            "seed": int(seed)}


def _prepare_knn(case, seed):
    N = 8  # the table needs the haplotypes only
    w = synth.Workload("small", N=N, S=case["S"], founders=20, depth=4.0, burnin=8, sampling=16)
    ch = synth_device.generate(w, N, case["S"], seed)
    haps = _host_words(_packed(_panel_bits(case["H"], case["S"], seed)))
    return {"eng": hmmlike.Engine(ch.emit.cpu().numpy(), ch.prob.cpu().numpy(), ch.tran, ch.pc,
                                  haps, 100)}


def _tally_haps(case, seed):
    return [_packed(_panel_bits(2 * case["N"], case["S"], 50 * seed + i, flips=0.02))
            for i in range(case["samples"])]


def _prepare_tally(case, seed):
    N, S = case["N"], case["S"]
    dev = hmmlike.HMMLikeCUDA(0)
    st = torch.cuda.Stream()
    dev._c(dev.L.glp_set_stream(dev.ctx, st.cuda_stream))
    haps = _tally_haps(case, seed)
    hsum = torch.zeros((2 * N, S), dtype=torch.int32, device="cuda")
    prob = torch.zeros((S, 2 * N), dtype=torch.float32, device="cuda")
    return {"dev": dev, "stream": st, "haps": haps, "hsum": hsum, "prob": prob}


def _prepare_codec(case, seed):
    ch = _chunk(case, seed)
    N, S = case["N"], case["S"]
    out = torch.zeros(((S + 7) // 8, N), dtype=torch.int32, device="cuda")
    return {"dev": hmmlike.HMMLikeCUDA(0), "gl": ch.prob, "out": out, "seed": int(seed)}


def _prepare_phase(case, seed):
    ch = _chunk(case, seed)
    r = np.full(case["S"], 2e-6)
    r[0] = 0.0
    m = model.Model(ch.prob[..., 1:3].contiguous().cpu().numpy(), r_morgans=r)
    opts = phase.PhaseOptions(sa_burnin=case["B"], burnin=case["I"], sampling=case["M"],
                              cycles=case["C"], seed=int(seed) + 1, knn=case["knn"],
                              cluster_start=3 if case["knn"] else 0,
                              recluster=case["recluster"], knn_metric=case["metric"])
    return {"model": m, "haps": _host_words(ch.haps), "opts": opts}


def prepare(case, seed):
    return dict({"generation": _prepare_generation, "batch": _prepare_batch,
                 "dropin": _prepare_dropin, "knn": _prepare_knn, "tally": _prepare_tally,
                 "codec": _prepare_codec, "phase": _prepare_phase}[case["kind"]](case, seed),
                case=case)


# ---------------------------------------------------------------------------
# one pass


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "generation":
        eng = state["eng"]
        a = eng.args(None, None, case["pen"], state["seed"], state["g"], neighbors=state["nbr"],
                     kick_first=case["panel"] > 0)
        state["g"] += 1
        eng.launch(a)
        eng.swap()
        eng.finish()
        return {"haps": eng.haps, "quad": eng.quad, "like": eng.like}
    if kind == "batch":
        state["batch"].run()
        dev = state["dev"]
        dev._c(dev.L.glp_finish(dev.ctx))
        return [{"haps": p.haps, "quad": p.quad, "like": p.like} for p in state["problems"]]
    if kind == "dropin":
        return state["dev"].run_hmm_on_device(state["panel"], state["props"], case["S"],
                                              case["N"], case["C"], state["quad"], state["seed"])
    if kind == "knn":
        nbr = state["eng"].knn(case["K"], metric=case["metric"])
        state["eng"].finish()
        return nbr
    if kind == "tally":
        dev, N, S = state["dev"], case["N"], case["S"]
        with torch.cuda.stream(state["stream"]):
            state["hsum"].zero_()
        for h in state["haps"]:
            dev._c(dev.L.glp_tally(dev.ctx, h.data_ptr(), N, S, state["hsum"].data_ptr()))
        dev._c(dev.L.glp_result(dev.ctx, state["hsum"].data_ptr(), N, S, case["samples"],
                                state["prob"].data_ptr()))
        dev._c(dev.L.glp_finish(dev.ctx))
        return {"hsum": state["hsum"], "prob": state["prob"]}
    if kind == "codec":
        dev, N, S = state["dev"], case["N"], case["S"]
        vq = glpack.GLVQ(state["gl"], np.random.default_rng(state["seed"]), device=dev)
        dev._c(dev.L.glp_vq_pack(dev.ctx, state["gl"].data_ptr(), N, S, vq.codebook.ctypes.data,
                                 16, 4, state["out"].data_ptr()))
        dev._c(dev.L.glp_finish(dev.ctx))
        return {"codebook": vq.codebook, "iterations": vq.iterations, "packed": state["out"]}
    prob, haps = phase.phase(state["model"], state["haps"], state["opts"])
    return {"prob": prob, "haps": haps.view(np.int64)}


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _generation_work(N, S, H, C, vq):
    """29 flops a site update of each of the C + 1 scored quadruples, and about
    80 a site of the haplotype sampling; emissions (or codes), genotype
    probabilities and haplotypes read once, the new haplotypes, quadruples and
    likelihoods written."""
    wn = (S + 63) // 64
    return {"bytes": N * S * (16 + 12 + (0.5 if vq else 0)) + 8 * wn * (H + 2 * N) + 24 * N +
            16 * S, "flops": 29.0 * N * (C + 1) * S + 80.0 * N * S}


def work(case):
    kind = case["kind"]
    if kind in ("generation", "phase"):
        w = _generation_work(case["N"], case["S"], 2 * case["N"] + case["panel"], case["C"],
                             case.get("vq", False))
        gens = case["B"] + case["I"] + case["M"] if kind == "phase" else 1
        return {k: v * gens for k, v in w.items()}
    if kind == "batch":
        ws = [_generation_work(N, S, 2 * N, case["C"], False)
              for N, S in _batch_shapes(case, 4)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    N, S = case.get("N", 0), case["S"]
    if kind == "dropin":
        wn = (S + 63) // 64
        return {"bytes": N * S / 2 + 16 * N * wn + 4 * N * (case["C"] + 8),
                "flops": 29.0 * N * (case["C"] + 1) * S}
    if kind == "knn":  # every unordered pair compared once, a compare and an add a site
        H, wn = case["H"], (S + 63) // 64
        return {"bytes": 8 * H * wn + 4 * (H // 2) * 2 * ((case["K"] + 1) // 2),
                "flops": float(H) * H * S}
    if kind == "tally":
        T = case["samples"]
        return {"bytes": T * (2 * N * ((S + 63) // 64) * 8 + 16 * N * S) + 16 * N * S,
                "flops": T * 6.0 * N * S + 2.0 * N * S}
    # codec: the GLs read once for the first codes, the codes written; 16 squared
    # distances a point for the assignment
    return {"bytes": 12.0 * N * S + N * S / 2, "flops": 16.0 * 5 * N * S}


# ---------------------------------------------------------------------------
# the same in 64 bits

_M32 = np.uint64(0xFFFFFFFF)


def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 (Salmon et al. 2011) on arrays of counters."""
    c = [np.asarray(v, dtype=np.uint64) for v in np.broadcast_arrays(c0, c1, c2, c3)]
    k0, k1 = np.uint64(seed & 0xFFFFFFFF), np.uint64(seed >> 32)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k0, p1 & _M32, (p0 >> np.uint64(32)) ^ c[3] ^ k1,
             p0 & _M32]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & _M32, (k1 + np.uint64(0xBB67AE85)) & _M32
    return c


def _uniform_hap(x, s, H):
    n = np.uint64(H - 2)
    h = ((x[0] << np.uint64(32)) | x[1]) % n
    return np.where(h >= 2 * s.astype(np.uint64), h + np.uint64(2), h).astype(np.int64)


def _loglik(emit, T, bits, quad):
    """log P of every sample's GLs given its quadruple: the product of the
    per-site matrices D_m T_m on the uniform start, as a balanced tree."""
    N, S = emit.shape[0], emit.shape[1]
    b = bits[quad].long()  # [4][N][S]
    states = torch.stack([2 * b[0] + b[2], 2 * b[0] + b[3], 2 * b[1] + b[2], 2 * b[1] + b[3]],
                         dim=-1)
    M = emit.gather(2, states)[..., None] * T[None]
    log = torch.zeros(N, dtype=torch.float64, device=emit.device)
    while M.shape[1] > 1:
        n = M.shape[1] // 2
        P = M[:, 1:2 * n:2] @ M[:, 0:2 * n:2]
        M = torch.cat([P, M[:, 2 * n:]], dim=1) if M.shape[1] % 2 else P
        top = M.amax(dim=(2, 3), keepdim=True)
        M = M / top
        log += top.log().sum(dim=(1, 2, 3))
    return log + (0.25 * M[:, 0].sum(dim=(1, 2))).log()


def _exact_generation(case, seed):
    N, S, C = case["N"], case["S"], case["C"]
    if case["vq"] or case["knn"] or case["panel"] or N * S * (C + 1) > 40_000_000:
        return None
    ch = _chunk(case, seed)
    H, s = ch.H, np.arange(N)
    emit = ch.emit.double()
    words = ch.haps
    bits = ((words[:, :, None] >> torch.arange(64, device="cuda")) & 1).reshape(H, -1)[:, :S]
    t = torch.from_numpy(ch.tran).double().cuda()
    t[0] = torch.tensor([1.0, 0.0, 0.0])
    T = torch.stack([t[:, [0, 1, 1, 2]], t[:, [1, 0, 2, 1]], t[:, [1, 2, 0, 1]],
                     t[:, [2, 1, 1, 0]]], dim=1)
    quad = torch.from_numpy(np.stack([_uniform_hap(_philox(j, s, 0, 3, seed), s, H)
                                      for j in range(4)])).cuda()
    curr = _loglik(emit, T, bits, quad)
    rows = torch.arange(N, device="cuda")
    for c in range(C):
        x = _philox(c, s, 0, 0, seed)
        slot = torch.from_numpy((x[0] & np.uint64(3)).astype(np.int64)).cuda()
        u = torch.from_numpy(((x[1] >> np.uint64(5)).astype(np.float64) * 67108864.0 +
                              (x[2] >> np.uint64(6)).astype(np.float64)) / 2.0**53).cuda()
        hap = torch.from_numpy(_uniform_hap(_philox(c, s, 0, 2, seed), s, H)).cuda()
        new = quad.clone()
        new[slot, rows] = hap
        prop = _loglik(emit, T, bits, new)
        take = (prop >= curr) | (u < ((prop - curr) * case["pen"]).exp())
        quad = torch.where(take[None, :], new, quad)
        curr = torch.where(take, prop, curr)
    return {"haps": None, "quad": None, "like": curr}


def _exact_tally(case, seed):
    N, S = case["N"], case["S"]
    hsum = torch.zeros((2 * N, S), dtype=torch.int32, device="cuda")
    at = torch.arange(64, device="cuda")
    for words in _tally_haps(case, seed):
        bits = torch.empty((2 * N, S), dtype=torch.int32, device="cuda")
        for i in range(0, 2 * N, 1000):
            bits[i:i + 1000] = ((words[i:i + 1000, :, None] >> at) & 1).reshape(
                -1, 64 * words.shape[1])[:, :S].int()
        a, b, x, y = bits[0::2], bits[1::2], hsum[0::2], hsum[1::2]
        keep = ((a * x + b * y).sum(dim=1) > (a * y + b * x).sum(dim=1))[:, None]
        first, second = torch.where(keep, a, b), torch.where(keep, b, a)
        hsum[0::2] += first
        hsum[1::2] += second
    return {"hsum": None, "prob": hsum.T.double() / case["samples"]}


def _splitmix64(x):
    """SplitMix64 (Steele, Lea, Flood 2014)."""
    x = (x + 0x9E3779B97F4A7C15) & (2**64 - 1)
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & (2**64 - 1)
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & (2**64 - 1)
    return x ^ (x >> 31)


def _exact_codec(case, seed):
    gl = _chunk(case, seed).prob.reshape(-1, 3)
    s = (gl[:, 0] + gl[:, 1]) + gl[:, 2]
    pts = torch.stack([gl[:, 0] / s, gl[:, 1] / s], dim=1).double()
    rng = np.random.default_rng(seed)
    rows = [(0.0, 1.0), (0.0, 0.0), (1.0, 0.0), (1.0 / 3, 1.0 / 3)]
    for _ in range(4, 16):
        a = float(np.float32(rng.random()))
        rows.append((a, float(np.float32(rng.random() * (1 - a)))))
    cb = torch.from_numpy(np.array(rows, dtype=np.float32)).double().cuda()

    def assign(cb):
        code, dist = [], 0.0
        for p in pts.split(1 << 21):
            d = (p[:, None, :] - cb[None]).square().sum(dim=2)
            code.append(d.argmin(dim=1))
            dist += float(d.amin(dim=1).sum())
        return torch.cat(code), dist

    seed_of_training = 0  # GLVQ's default
    code, cur = assign(cb)
    prev, it = float("inf"), 0
    while abs(cur - prev) > cur / 100 and it < 1000:
        it, prev = it + 1, cur
        n = torch.bincount(code, minlength=16)
        cb = torch.stack([torch.bincount(code, weights=pts[:, j], minlength=16) / n
                          for j in range(2)], dim=1)
        for k in (n == 0).nonzero().flatten().tolist():  # moves onto a drawn point
            cb[k] = pts[_splitmix64(seed_of_training ^ ((it << 16) | k)) % len(pts)]
        code, cur = assign(cb)
    return {"codebook": cb, "iterations": None, "packed": None}


def exact(case, seed):
    fn = {"generation": _exact_generation, "tally": _exact_tally,
          "codec": _exact_codec}.get(case["kind"])
    return fn(case, int(seed)) if fn else None
