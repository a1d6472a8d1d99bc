"""Timing cases of the candidate-verification library, through its public entry points.

A case is a dict of plain values; `listed` gives the fixed ones, `draw` more of the same
ranges, `prepare` builds a case's inputs and context from a seed, `run` makes one call.
Workloads are synthetic with the shapes of `kira_ls_aligner_b200.synth` (uniform
reference with 300 bp repeat families, reads with substitutions and indels, one true
candidate window per read), generated on the GPU so that a preparation is quick.

Kinds of calls:
  verify_dev   kira_gpu_verify_dev: sieve, certificate, Myers and banded SW on
               device-resident pairs over a resident reference
  verify_host  kira_gpu_verify_batch_compact: the same cascade from pinned host buffers
  bsw          kira_gpu_bsw_batch: banded SW with CIGAR from host buffers (windows from
               the resident reference), bands drawn per pair
  wfa          kira_gpu_wfa_batch: the cascade's wavefront step from host buffers
  prefilter    kira_gpu_prefilter_batch: stage 4's exact match + ungapped prefilter
  simd         kira_gpu_align_batch_simd: full-window batch SW on host windows
  sieve        kira_gpu_sieve_batch: the packed multi-shift scan on host jobs
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from kira_ls_aligner_b200 import (AlignmentConfig, GpuContext, PairBatch, PrefilterConfig,
                                  VerifyParams, WfaParams, _abi, autotune)

SLACK = 100  # window bases beyond the read in the verification workloads


def listed() -> list:
    return [
        # One worker's call with a handful of reads: latency and launches.
        dict(name="verify_64", kind="verify_dev", reads=16, cands=4, q_lo=150, q_hi=150, band=33,
             router=False, n_bases=False, ref_len=1_000_000, tuned=False),
        # The small configuration: 10k reads x 4 windows on 1 Mbp.
        dict(name="verify_40k", kind="verify_dev", reads=10_000, cands=4, q_lo=150, q_hi=150,
             band=33, router=False, n_bases=False, ref_len=1_000_000, tuned=False),
        # A serving request: reads of U[100, 250] bp, ambiguous bases, the router's own
        # thresholds (which send most pairs through Myers).
        dict(name="verify_mixed_131k", kind="verify_dev", reads=32_768, cands=4, q_lo=100,
             q_hi=250, band=33, router=True, n_bases=True, ref_len=20_000_000, tuned=False),
        # The batched configuration: 2M pairs of 150 / 250 bp, launch shape autotuned
        # once as the benchmark does.
        dict(name="verify_2m", kind="verify_dev", reads=250_000, cands=8, q_lo=150, q_hi=150,
             band=33, router=False, n_bases=False, ref_len=100_000_000, tuned=True),
        # The same batch end to end from pinned host memory, with the compact results.
        dict(name="verify_host_2m", kind="verify_host", reads=250_000, cands=8, q_lo=150,
             q_hi=150, band=33, router=False, n_bases=False, ref_len=100_000_000, tuned=False),
        # Uneven-length batch: reads U[50, 300], bands 16 to 128.
        dict(name="bsw_uneven_500k", kind="bsw", pairs=500_000, q_lo=50, q_hi=300, band_lo=16,
             band_hi=128, err_lo=0.0, err_hi=0.03, indels=0.2, ref_len=20_000_000),
        # Long-read gap-fill segments, band 256: a full batch, and a request of a few reads.
        dict(name="bsw_gapfill_20k", kind="bsw", pairs=20_000, q_lo=200, q_hi=2000, band_lo=256,
             band_hi=256, err_lo=0.05, err_hi=0.12, indels=0.5, ref_len=20_000_000),
        dict(name="bsw_gapfill_50", kind="bsw", pairs=50, q_lo=200, q_hi=2000, band_lo=256,
             band_hi=256, err_lo=0.05, err_hi=0.12, indels=0.5, ref_len=20_000_000),
        # The cascade's WFA step with traceback, scored costs and router budget.
        dict(name="wfa_1m", kind="wfa", pairs=1_000_000, q_lo=150, q_hi=150, slack=33,
             err_hi=0.04, scored=True, traceback=True, ref_len=20_000_000),
        # Stage 4's exact match + prefilter over one contig.
        dict(name="prefilter_400k", kind="prefilter", pairs=400_000, q_lo=150, q_hi=150,
             ref_len=20_000_000),
        # Full-window batch SW (the SIMD batch drop-in), one read and window length per call.
        dict(name="simd_4k", kind="simd", pairs=4096, q_lo=150, q_hi=150, slack=SLACK,
             ref_len=1_000_000),
        # The GPU sieve drop-in on packed host jobs.
        dict(name="sieve_20k", kind="sieve", pairs=20_000, q_lo=150, q_hi=150, slack=SLACK,
             ref_len=1_000_000),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["verify_dev"] * 4 + ["verify_host"] * 2 + ["bsw"] * 3 + ["gapfill"] * 2 +
                      ["wfa"] * 2 + ["prefilter", "simd", "sieve"])
    if kind in ("verify_dev", "verify_host"):
        q_lo = rng.choice([100, 125, 150, 151, rng.randint(60, 200)])
        q_hi = rng.choice([q_lo, q_lo, min(250, q_lo + rng.randint(1, 150))])
        return dict(kind=kind, reads=_log_int(rng, 16, 180_000), cands=rng.randint(1, 8), q_lo=q_lo,
                    q_hi=q_hi, band=rng.choice([33, 33, 33, 20, 50]), router=rng.random() < 0.4,
                    n_bases=rng.random() < 0.5, ref_len=rng.choice([1_000_000, 20_000_000]),
                    tuned=False)
    if kind == "bsw":
        q_lo = rng.randint(40, 150)
        b = rng.choice([16, 24, 33, 64])
        return dict(kind="bsw", pairs=_log_int(rng, 50, 400_000), q_lo=q_lo,
                    q_hi=q_lo + rng.randint(0, 150), band_lo=b, band_hi=b * rng.choice([1, 2]),
                    err_lo=0.0, err_hi=0.03, indels=0.2, ref_len=20_000_000)
    if kind == "gapfill":
        q_lo = rng.randint(150, 600)
        b = rng.choice([128, 200, 256])
        return dict(kind="bsw", pairs=_log_int(rng, 50, 16_000), q_lo=q_lo,
                    q_hi=q_lo + rng.randint(100, 1400), band_lo=b, band_hi=b, err_lo=0.05,
                    err_hi=0.12, indels=0.5, ref_len=20_000_000)
    if kind == "wfa":
        q_lo = rng.randint(75, 200)
        return dict(kind="wfa", pairs=_log_int(rng, 1000, 700_000), q_lo=q_lo,
                    q_hi=q_lo + rng.choice([0, rng.randint(1, 50)]), slack=rng.randint(16, 48),
                    err_hi=rng.choice([0.02, 0.04]), scored=rng.random() < 0.7,
                    traceback=rng.random() < 0.7, ref_len=20_000_000)
    if kind == "prefilter":
        q_lo = rng.randint(75, 200)
        return dict(kind="prefilter", pairs=_log_int(rng, 1000, 400_000), q_lo=q_lo,
                    q_hi=q_lo + rng.choice([0, rng.randint(1, 50)]), ref_len=20_000_000)
    q = rng.randint(60, 250)
    return dict(kind=kind, pairs=_log_int(rng, 32, 4096 if kind == "simd" else 20_000), q_lo=q,
                q_hi=q, slack=rng.randint(20, 120), ref_len=1_000_000)


# --- inputs ----------------------------------------------------------------------
DEV = "cuda"
_BASES = {}


def _acgt() -> torch.Tensor:
    if "t" not in _BASES:
        _BASES["t"] = torch.tensor([65, 67, 71, 84], dtype=torch.uint8, device=DEV)
    return _BASES["t"]


def _uniform(g, n, lo, hi):
    return torch.rand(n, generator=g, device=DEV) * (hi - lo) + lo


def _ints(g, n, lo, hi):
    """n integers of [lo, hi]."""
    return torch.randint(lo, hi + 1, (n,), generator=g, device=DEV)


def _reference(g, length: int) -> torch.Tensor:
    """ASCII bases, 5 % of them copies (2-10 % diverged) of 200 families of 300 bp."""
    code = torch.randint(0, 4, (length,), generator=g, device=DEV, dtype=torch.uint8)
    slots = length // 300
    k = slots // 20
    at = torch.randperm(slots, generator=g, device=DEV)[:k]
    fam = torch.randint(0, 4, (200, 300), generator=g, device=DEV, dtype=torch.uint8)
    rep = fam[_ints(g, k, 0, 199)]
    div = torch.rand((k, 300), generator=g, device=DEV) < _uniform(g, k, 0.02, 0.10)[:, None]
    rep = (rep + div * torch.randint(1, 4, (k, 300), generator=g, device=DEV,
                                     dtype=torch.uint8)) % 4
    code[: slots * 300].view(slots, 300)[at] = rep
    return _acgt()[code.long()] if length <= 20_000_000 else torch.cat(
        [_acgt()[c.long()] for c in code.split(20_000_000)])


def _simulate(g, ref, origin, q, rate, sub, ins, n_bases=False):
    """Reads of q bases drawn from ref at origin with per-read error rate `rate`, split
    into the shares sub, ins and the rest deletions. Returns (flat bases, offsets)."""
    n, qm = int(q.numel()), int(q.max())
    parts = []
    for a in range(0, n, 32_768):
        b = min(n, a + 32_768)
        u = torch.rand((b - a, qm), generator=g, device=DEV)
        r = rate[a:b, None]
        is_sub = u < r * sub
        is_ins = (u >= r * sub) & (u < r * (sub + ins))
        is_del = (u >= r * (sub + ins)) & (u < r)
        adv = 1 - is_ins.int() + is_del.int()
        src = torch.cumsum(adv, 1) - adv + is_del.int()
        bases = ref[(origin[a:b, None] + src).clamp_(max=ref.numel() - 1)]
        rnd = torch.randint(0, 4, (b - a, qm), generator=g, device=DEV, dtype=torch.uint8)
        code = ((bases >> 1) ^ (bases >> 2)) & 3  # A0 C1 G2 T3
        code = torch.where(is_sub, (code + 1 + rnd % 3) % 4, torch.where(is_ins, rnd, code))
        bases = _acgt()[code.long()]
        if n_bases:
            bases[torch.rand((b - a, qm), generator=g, device=DEV) < 2e-4] = 78  # N
        parts.append(bases[torch.arange(qm, device=DEV)[None, :] < q[a:b, None]])
    off = torch.cumsum(q, 0) - q
    return torch.cat(parts), off


def _pinned(t: torch.Tensor) -> np.ndarray:
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _pinned_empty(n: int, dtype=np.uint8) -> np.ndarray:
    return torch.zeros(n * np.dtype(dtype).itemsize, dtype=torch.uint8,
                       pin_memory=True).numpy().view(dtype)


def _pad(t: torch.Tensor) -> torch.Tensor:
    return torch.cat([t, torch.zeros(16, dtype=torch.uint8, device=DEV)])


def _verify_pairs(case, g, ref):
    n, c = case["reads"], case["cands"]
    q = _ints(g, n, case["q_lo"], case["q_hi"])
    qm = case["q_hi"]
    origin = _ints(g, n, SLACK, ref.numel() - 2 * qm - SLACK)
    rate = _uniform(g, n, 0.006, 0.021)  # substitutions U[0.5 %, 2 %] plus 0.1 % indels
    reads, off = _simulate(g, ref, origin, q, rate, 0.92, 0.04, case["n_bases"])
    win_off = _ints(g, n * c, 0, ref.numel() - qm - SLACK - 1)
    lead = _ints(g, n, 0, SLACK)
    true = torch.arange(n, device=DEV) * c + _ints(g, n, 0, c - 1)
    win_off[true] = origin - lead
    rep = lambda t: t.repeat_interleave(c)  # noqa: E731
    return reads, rep(off), rep(q).int(), win_off, rep(q + SLACK).int()


def prepare(case: dict, seed: int) -> dict:
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 1_000_003 + 17)
    ref = _reference(g, case["ref_len"])
    ctx = GpuContext(0)
    if case["kind"] not in ("simd", "sieve"):
        ctx.ref_upload(ref.cpu().numpy())
    s = {"kind": case["kind"], "ctx": ctx, "L": _abi.lib()}
    _PREPARE[case["kind"]](case, g, ref, s)
    torch.cuda.synchronize()
    return s


def _params(case) -> VerifyParams:
    cfg = AlignmentConfig(bandwidth=case["band"])
    return VerifyParams(cfg, -1, -1) if case["router"] else VerifyParams(cfg, 12, 8)


def _prepare_verify_dev(case, g, ref, s):
    reads, roff, rlen, woff, wlen = _verify_pairs(case, g, ref)
    n = int(roff.numel())
    s["keep"] = [_pad(reads), roff.contiguous(), rlen.contiguous(), woff.contiguous(),
                 wlen.contiguous()]
    p = _abi.Pairs()
    p.n, p.max_read_len, p.max_win_len = n, case["q_hi"], case["q_hi"] + SLACK
    p.read_seq, p.read_seq_bytes = s["keep"][0].data_ptr(), int(reads.numel())
    p.read_off, p.read_len, p.win_off, p.win_len = [t.data_ptr() for t in s["keep"][1:]]
    p.win_seq = None
    s["pairs"], s["params"] = p, _params(case).to_c()
    s["cap"] = max(64, 2 * n)
    s["rows"] = torch.zeros(8 * n, dtype=torch.int32, device=DEV)
    s["ops"] = torch.zeros(s["cap"], dtype=torch.int32, device=DEV)
    s["used"] = torch.zeros(1, dtype=torch.int64, device=DEV)
    if case["tuned"]:
        def once():
            _run_verify_dev(s)
            torch.cuda.synchronize()
        autotune.tune_bsw_shape(s["ctx"], case["band"], once, repeats=2,
                                device_name=torch.cuda.get_device_name(0))


def _run_verify_dev(s):
    stream = torch.cuda.current_stream().cuda_stream
    s["ctx"].check(s["L"].kira_gpu_verify_dev(
        s["ctx"].handle, C.byref(s["pairs"]), C.byref(s["params"]), s["rows"].data_ptr(),
        s["ops"].data_ptr(), s["cap"], s["used"].data_ptr(), None, None, C.c_void_p(stream)))
    return [s["rows"], s["ops"], s["used"]]


def _prepare_verify_host(case, g, ref, s):
    reads, roff, rlen, woff, wlen = _verify_pairs(case, g, ref)
    n = int(roff.numel())
    s["batch"] = PairBatch(_pinned(_pad(reads)), _pinned(roff).view(np.uint64),
                           _pinned(rlen).view(np.uint32), None, _pinned(woff).view(np.uint64),
                           _pinned(wlen).view(np.uint32))
    s["pairs"], s["params"] = s["batch"].to_c(), _params(case).to_c()
    s["status"], s["rows"] = _pinned_empty(n), _pinned_empty(8 * n, np.int32)
    s["ops"] = _pinned_empty(max(64, 2 * n), np.int32)
    s["n"] = n


def _run_verify_host(s):
    cb = _abi.CigarBuf(s["ops"].ctypes.data, len(s["ops"]), 0)
    rows, cells = C.c_uint64(), C.c_uint64()
    s["ctx"].check(s["L"].kira_gpu_verify_batch_compact(
        s["ctx"].handle, C.byref(s["pairs"]), C.byref(s["params"]), s["status"].ctypes.data,
        s["rows"].ctypes.data, s["n"], C.byref(rows), C.byref(cb), C.byref(cells)))
    return [s["status"], s["rows"], s["ops"], int(rows.value), int(cb.used), int(cells.value)]


def _prepare_bsw(case, g, ref, s):
    n = case["pairs"]
    q = _ints(g, n, case["q_lo"], case["q_hi"])
    octaves = int(round(math.log2(case["band_hi"] / case["band_lo"])))
    band = case["band_lo"] * 2 ** _ints(g, n, 0, octaves)
    start = _ints(g, n, 0, ref.numel() - 2 * case["q_hi"] - 2 * case["band_hi"] - 512)
    rate = _uniform(g, n, case["err_lo"], case["err_hi"])
    reads, off = _simulate(g, ref, start + band, q, rate, 1.0 - case["indels"],
                           case["indels"] / 2)
    band = band.int()
    s["batch"] = PairBatch(_pinned(_pad(reads)), _pinned(off).view(np.uint64),
                           _pinned(q.int()).view(np.uint32), None, _pinned(start).view(np.uint64),
                           _pinned((q + 2 * band).int()).view(np.uint32), _pinned(band), None,
                           _pinned(band))
    s["cfg"] = AlignmentConfig()
    s["pairs"], s["cc"] = s["batch"].to_c(), s["cfg"].to_c()
    s["rows"] = _pinned_empty(8 * n, np.int32)
    s["ops"] = _pinned_empty(max(16, 8 * n, n * case["q_hi"] // 4), np.int32)
    # A program with a steady batch keeps its launches as a graph.
    s["ctx"].check(s["L"].kira_gpu_set_graphs(s["ctx"].handle, 1, None, None))


def _run_bsw(s):
    cb = _abi.CigarBuf(s["ops"].ctypes.data, len(s["ops"]), 0)
    cells = C.c_uint64()
    s["ctx"].check(s["L"].kira_gpu_bsw_batch(s["ctx"].handle, C.byref(s["pairs"]),
                                             C.byref(s["cc"]), s["rows"].ctypes.data,
                                             C.byref(cb), C.byref(cells)))
    return [s["rows"], s["ops"], int(cb.used), int(cells.value)]


def _prepare_wfa(case, g, ref, s):
    n = case["pairs"]
    q = _ints(g, n, case["q_lo"], case["q_hi"])
    start = _ints(g, n, 0, ref.numel() - 2 * case["q_hi"] - case["slack"] - 64)
    reads, off = _simulate(g, ref, start, q, _uniform(g, n, 0.0, case["err_hi"]), 4 / 6, 1 / 6)
    s["batch"] = PairBatch(_pinned(_pad(reads)), _pinned(off).view(np.uint64),
                           _pinned(q.int()).view(np.uint32), None, _pinned(start).view(np.uint64),
                           _pinned((q + case["slack"]).int()).view(np.uint32))
    cfg = AlignmentConfig()
    w = (WfaParams.scored_from(cfg, traceback=case["traceback"]) if case["scored"] else
         WfaParams(cfg.mismatch, cfg.gap_open, cfg.gap_extend, traceback=case["traceback"]))
    s["pairs"], s["params"] = s["batch"].to_c(), w.to_c()
    s["rows"], s["ops"] = _pinned_empty(8 * n, np.int32), _pinned_empty(8 * n, np.int32)


def _run_wfa(s):
    cb = _abi.CigarBuf(s["ops"].ctypes.data, len(s["ops"]), 0)
    s["ctx"].check(s["L"].kira_gpu_wfa_batch(s["ctx"].handle, C.byref(s["pairs"]),
                                             C.byref(s["params"]), None, None,
                                             s["rows"].ctypes.data, C.byref(cb)))
    return [s["rows"], s["ops"], int(cb.used)]


def _prepare_prefilter(case, g, ref, s):
    n = case["pairs"]
    q = _ints(g, n, case["q_lo"], case["q_hi"])
    origin = _ints(g, n, 64, ref.numel() - 2 * case["q_hi"] - 128)
    exact = torch.rand(n, generator=g, device=DEV) < 0.3
    rate = torch.where(exact, torch.zeros(n, device=DEV), _uniform(g, n, 0.0, 0.02))
    reads, off = _simulate(g, ref, origin, q, rate, 0.8, 0.1)
    lo = torch.where(exact, 0, _ints(g, n, 0, 39))
    hi = torch.where(exact, q, q - _ints(g, n, 0, 34))
    lo = torch.minimum(lo, hi - 1)
    sign = 2 * _ints(g, n, 0, 1) - 1
    skew = torch.where(torch.rand(n, generator=g, device=DEV) < 0.1, _ints(g, n, 1, 3) * sign, 0)
    skew = torch.maximum(skew, lo - hi + 1)
    rs = origin + lo
    chains = torch.stack([rs, rs + (hi - lo) + skew, lo, hi], 1).int()
    s["batch"] = PairBatch(_pinned(_pad(reads)), _pinned(off).view(np.uint64),
                           _pinned(q.int()).view(np.uint32), None,
                           _pinned_empty(n, np.uint64),
                           _pinned(torch.full_like(q, ref.numel()).int()).view(np.uint32))
    s["chains"] = _pinned(chains)
    s["top1"] = _pinned((torch.rand(n, generator=g, device=DEV) < 0.9).to(torch.uint8))
    s["margin"] = _pinned(_ints(g, n, -5, 39).int())
    s["pairs"], s["params"] = s["batch"].to_c(), PrefilterConfig().to_c()
    s["rows"] = _pinned_empty(12 * n, np.int32)
    s["ops"], s["md"] = _pinned_empty(3 * n + 16, np.int32), _pinned_empty(16 * n + 64)


def _run_prefilter(s):
    cb = _abi.CigarBuf(s["ops"].ctypes.data, len(s["ops"]), 0)
    used = C.c_uint64()
    s["ctx"].check(s["L"].kira_gpu_prefilter_batch(
        s["ctx"].handle, C.byref(s["pairs"]), s["chains"].ctypes.data, s["top1"].ctypes.data,
        s["margin"].ctypes.data, C.byref(s["params"]), s["rows"].ctypes.data, C.byref(cb),
        s["md"].ctypes.data, len(s["md"]), C.byref(used)))
    return [s["rows"], s["ops"], s["md"], int(cb.used), int(used.value)]


def _read_windows(case, g, ref):
    """Reads of q bases against windows of q + slack with the read's origin inside."""
    n, q, w = case["pairs"], case["q_lo"], case["q_lo"] + case["slack"]
    start = _ints(g, n, 0, ref.numel() - w - q - 1)
    lead = _ints(g, n, 0, case["slack"])
    ql = torch.full((n,), q, device=DEV)
    reads, off = _simulate(g, ref, start + lead, ql, _uniform(g, n, 0.0, 0.04), 0.8, 0.1)
    return reads, off, ref[start[:, None] + torch.arange(w, device=DEV)[None, :]]


def _prepare_simd(case, g, ref, s):
    reads, off, wins = _read_windows(case, g, ref)
    n, w = int(wins.shape[0]), int(wins.shape[1])
    s["batch"] = PairBatch(_pinned(_pad(reads)), _pinned(off).view(np.uint64),
                           np.full(n, case["q_lo"], np.uint32), _pinned(_pad(wins.reshape(-1))),
                           np.arange(n, dtype=np.uint64) * np.uint64(w), np.full(n, w, np.uint32))
    s["pairs"], s["cc"] = s["batch"].to_c(), AlignmentConfig().to_c()
    s["rows"], s["ops"] = _pinned_empty(8 * n, np.int32), _pinned_empty(8 * n + 16, np.int32)


def _run_simd(s):
    cb = _abi.CigarBuf(s["ops"].ctypes.data, len(s["ops"]), 0)
    s["ctx"].check(s["L"].kira_gpu_align_batch_simd(  # AVX2 requested and found
        s["ctx"].handle, C.byref(s["pairs"]), C.byref(s["cc"]), 1, 1, s["rows"].ctypes.data,
        C.byref(cb)))
    return [s["rows"], s["ops"], int(cb.used)]


_JOB = np.dtype([("read", "<u8"), ("read_bytes", "<u4"), ("read_nucs", "<u4"), ("win", "<u8"),
                 ("win_bytes", "<u4"), ("win_nucs", "<u4"), ("max_mism", "<u4"), ("pad", "<u4")])
assert _JOB.itemsize == C.sizeof(_abi.SieveJob)


def _pack2(bases: torch.Tensor) -> np.ndarray:
    """Rows of ASCII bases as rows of 2-bit packed bytes."""
    code = ((bases >> 1) ^ (bases >> 2)) & 3
    code = torch.nn.functional.pad(code, (0, -code.shape[1] % 4)).view(code.shape[0], -1, 4)
    return (code[..., 0] | code[..., 1] << 2 | code[..., 2] << 4 | code[..., 3] << 6).cpu().numpy()


def _prepare_sieve(case, g, ref, s):
    reads, _, wins = _read_windows(case, g, ref)
    n, q = case["pairs"], case["q_lo"]
    s["reads"], s["wins"] = _pack2(reads.view(n, q)), _pack2(wins)
    jobs = np.zeros(n, _JOB)
    for key, a, nucs in (("read", s["reads"], q), ("win", s["wins"], int(wins.shape[1]))):
        jobs[key] = a.ctypes.data + np.arange(n, dtype=np.uint64) * np.uint64(a.shape[1])
        jobs[key + "_bytes"], jobs[key + "_nucs"] = a.shape[1], nucs
    jobs["max_mism"] = 12
    s["jobs"], s["n"] = jobs, n
    s["out"] = np.zeros((n, 3), np.int32)


def _run_sieve(s):
    s["ctx"].check(s["L"].kira_gpu_sieve_batch(
        s["ctx"].handle, C.cast(s["jobs"].ctypes.data, C.POINTER(_abi.SieveJob)), s["n"],
        C.cast(s["out"].ctypes.data, C.POINTER(_abi.SieveResult))))
    return s["out"]


_PREPARE = {"verify_dev": _prepare_verify_dev, "verify_host": _prepare_verify_host,
            "bsw": _prepare_bsw, "wfa": _prepare_wfa, "prefilter": _prepare_prefilter,
            "simd": _prepare_simd, "sieve": _prepare_sieve}
_RUN = {"verify_dev": _run_verify_dev, "verify_host": _run_verify_host, "bsw": _run_bsw,
        "wfa": _run_wfa, "prefilter": _run_prefilter, "simd": _run_simd, "sieve": _run_sieve}


def run(state: dict):
    """One call. Outputs are the caller's buffers (rows, CIGAR ops and text, zero past what
    the call wrote) and the counts it reports."""
    return _RUN[state["kind"]](state)


# --- work ------------------------------------------------------------------------
# Integer operations of the reference's recurrences: a banded-SW cell 18
# (src/alignment/mod.rs:1462-1539), a Myers column word 10, a sieve word per shift 6.
SW_OPS, MYERS_OPS, SIEVE_OPS = 18, 10, 6


def work(case: dict) -> dict:
    q = (case["q_lo"] + case["q_hi"]) / 2
    kind = case["kind"]
    if kind in ("verify_dev", "verify_host"):
        n = case["reads"] * case["cands"]
        # Reads once, each window once, 24 B of descriptors, a 32-byte row a pair (the
        # compact form: a status byte, and rows for the true pairs).
        out = 32 * n if kind == "verify_dev" else n + 36 * case["reads"]
        nbytes = case["reads"] * q + n * (q + SLACK + 24) + out
        # The true pair of every read is sieved, and about 0.4 of them are aligned.
        ops = case["reads"] * (SIEVE_OPS * (SLACK + 1) * q / 32 +
                               0.4 * SW_OPS * q * (2 * case["band"] + 1))
        if case["router"]:
            ops += n * MYERS_OPS * (q + SLACK) * q / 32
        return {"bytes": nbytes, "flops": ops}
    n = case["pairs"]
    if kind == "bsw":
        octaves = int(round(math.log2(case["band_hi"] / case["band_lo"])))
        band = sum(case["band_lo"] * 2 ** k for k in range(octaves + 1)) / (octaves + 1)
        # Reads, windows, 32 B of descriptors, rows and CIGARs; half a byte of trace a cell.
        cells = n * q * (2 * band + 1)
        return {"bytes": n * (2 * q + 2 * band + 32 + 32 + 16), "flops": SW_OPS * cells}
    if kind == "wfa":
        # Mean cost about 0.12 per base at 4 % errors; 3 x (cost + 1) x about 12 cells.
        return {"bytes": n * (2 * q + case["slack"] + 24 + 32 + 12), "flops": n * 36 * q * 0.12}
    if kind == "prefilter":
        return {"bytes": n * (2 * q + 24 + 16 + 5 + 48 + 16), "flops": n * 4 * q}
    w = q + case["slack"]
    if kind == "simd":
        return {"bytes": n * (q + w + 24 + 32 + 12), "flops": n * SW_OPS * q * w}
    return {"bytes": n * (q / 4 + w / 4 + 40 + 12),
            "flops": n * SIEVE_OPS * (case["slack"] + 1) * q / 32}


def exact(case: dict, seed: int):
    """Every output is a whole number (scores, coordinates, CIGAR ops, text bytes), which
    has to be equal: there is no rounding to hold against 64 bits."""
    return None
