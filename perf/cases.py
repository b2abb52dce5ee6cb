"""Workloads of the dedispersion search path, for timing it and comparing its results.

Each case is one call (or one pass of calls) that a search pipeline makes: ingest of raw spectra,
RFI clip, brute-force and two-stage subband dedispersion, single-pulse detection, and the batched
form.  `listed` holds the cases with their sizes; `draw` gives more cases over the same ranges.
The band is 300 MHz below 1500 MHz at 64 us unless a case says otherwise.
"""
import math

import numpy as np
import torch

import mdsm_gb300 as m
from mdsm_gb300 import sigproc
from mdsm_gb300.batch import Batch

FCH1, BW, TSAMP = 1500.0, 300.0, 64e-6
K_PLAN = 4148.741601   # the plans' dispersion constant
K_PULSE = 4148.808     # the injected pulses' dispersion constant
THRESHOLD = 6.0
SLOTS = 4096           # candidates of a list that `run` returns
_ELEM = {"u8": 1, "u16": 2, "i16": 2, "f32": 4}
_TORCH = {"u8": torch.uint8, "u16": torch.uint16, "i16": torch.int16, "f32": torch.float32}


def listed():
    return [
        # The smallest brute-force call: one short block of a narrow DM range, as a monitor of one
        # known source makes for every block; launch and call costs count.
        dict(name="brute_u8_small", kind="brute", dtype="u8", nchans=512, nsamp=4096, ndms=76,
             lowdm=0.0, dmstep=0.5, steps=1, bw=300.0),
        # Float samples, 256 channels x 32768 samples in, 500 trials: the plain path at the size
        # that a workstation runs.
        dict(name="brute_f32_256ch", kind="brute", dtype="f32", nchans=256, nsamp=32344, ndms=500,
             lowdm=0.0, dmstep=0.2, steps=1, bw=100.0),
        # 16-bit samples at the high-DM end with coarse steps, ragged in samples and trials.
        dict(name="brute_i16_ragged", kind="brute", dtype="i16", nchans=2048, nsamp=30011,
             ndms=517, lowdm=400.0, dmstep=0.9765625, steps=1, bw=300.0),
        # The full band: 4096 channels, 2^18 samples, 4096 trials 0-2000 with the step doubling at
        # 500 and 1000.  The largest call.
        dict(name="brute_u8_full", kind="brute", dtype="u8", nchans=4096, nsamp=262144, ndms=4096,
             lowdm=0.0, dmstep=0.244140625, steps=3, bw=300.0),
        # The same trials by the two-stage subband method on one block of a many-beam server.
        dict(name="subband_u8_block", kind="subband", dtype="u8", nchans=4096, nsubs=64,
             nsamp=65536, ncalls=128, calldms=16, dmstep=0.244140625, npasses=3, bin0=1),
        # Float samples with passes downsampled by 1, 2 and 4, as a planner for a survey gives them.
        dict(name="subband_f32_downsampled", kind="subband", dtype="f32", nchans=1024, nsubs=32,
             nsamp=32768, ncalls=32, calldms=16, dmstep=0.5, npasses=3, bin0=2),
        # RFI clip of a server's 8-bit block, before every dedispersion.
        dict(name="clip_u8_block", kind="clip", dtype="u8", nchans=4096, nsamp=97921),
        # RFI clip of a float block with ragged sizes.
        dict(name="clip_f32_ragged", kind="clip", dtype="f32", nchans=1001, nsamp=40003),
        # Boxcar search of a block's exact integer series, nine widths.
        dict(name="boxcar_i32_block", kind="boxcar", dtype="i32", ndms=4096, nsamp=65536,
             nwidths=9),
        # The reference's detector (block statistics, median of five) on float series.
        dict(name="detect_f32_block", kind="detect", dtype="f32", ndms=1024, nsamp=65536),
        # Ingest: 8-bit time-major spectra to the channel-major block.
        dict(name="ingest_8bit_block", kind="ingest", nbits=8, out="u8", nchans=4096,
             nsamp=65536, invert=False),
        # The batched form: uneven beams clipped, dedispersed and searched as one pass.
        dict(name="batch_4beams", kind="batch", nbeams=4, nsamp=16384, spread=4, nchans=1024,
             ndms=1024, maxdm=900.0),
    ]


def _log(rng, lo, hi):
    """A whole number spread over [lo, hi] by its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["brute", "brute", "brute", "subband", "subband", "clip", "clip", "boxcar",
                       "detect", "ingest", "batch"])
    if kind == "brute":
        dtype = rng.choice(["u8", "u8", "i16", "f32"])
        while True:
            c = dict(kind=kind, dtype=dtype, nchans=_log(rng, 64, 4096),
                     nsamp=_log(rng, 2000, 262144), ndms=_log(rng, 32, 4096),
                     lowdm=round(rng.choice([0.0, rng.uniform(0, 400)]), 3),
                     dmstep=round(math.exp(rng.uniform(math.log(0.2), math.log(1.0))), 4),
                     steps=rng.choice([1, 1, 3]), bw=rng.choice([100.0, 300.0]))
            cost = c["nchans"] * c["nsamp"] * c["ndms"]
            if cost <= (5e11 if dtype == "u8" else 5e10):
                return c
    if kind == "subband":
        nchans = rng.choice([512, 1024, 2048, 4096])
        return dict(kind=kind, dtype=rng.choice(["u8", "u8", "f32"]), nchans=nchans,
                    nsubs=rng.choice([32, 64]), nsamp=4 * _log(rng, 512, 16384),
                    ncalls=_log(rng, 4, 64), calldms=rng.choice([8, 16, 16, 24, 32]),
                    dmstep=rng.choice([0.25, 0.5, 1.0]), npasses=rng.choice([1, 2, 3]),
                    bin0=rng.choice([1, 2]))
    if kind == "clip":
        return dict(kind=kind, dtype=rng.choice(["u8", "i16", "f32"]),
                    nchans=_log(rng, 64, 4096), nsamp=_log(rng, 2000, 97921))
    if kind == "boxcar":
        return dict(kind=kind, dtype=rng.choice(["i32", "f32"]), ndms=_log(rng, 16, 4096),
                    nsamp=_log(rng, 1000, 65536), nwidths=rng.choice([5, 7, 9]))
    if kind == "detect":
        return dict(kind=kind, dtype="f32", ndms=_log(rng, 16, 1024), nsamp=_log(rng, 1000, 65536))
    if kind == "ingest":
        nbits = rng.choice([2, 4, 8, 8, 16, 32])
        out = {16: rng.choice(["u16", "i16", "f32"]), 32: "f32"}.get(nbits, rng.choice(["u8", "f32"]))
        return dict(kind=kind, nbits=nbits, out=out, nchans=4 * _log(rng, 16, 1024),
                    nsamp=_log(rng, 1000, 65536), invert=rng.random() < 0.5)
    return dict(kind=kind, nbeams=rng.randint(1, 4), nsamp=_log(rng, 4096, 16384),
                spread=rng.choice([1, 2, 4]), nchans=rng.choice([512, 1024]),
                ndms=32 * rng.randint(8, 32), maxdm=round(rng.uniform(200, 900), 2))


# ---- the plans' shifts, restated in numpy for `exact` and `work` --------------------------------

def _segments(case):
    """(lowdm, dmstep, ndms) runs; three runs double the step twice, half and a quarter of the
    trials each."""
    n, lo, st = case["ndms"], case["lowdm"], case["dmstep"]
    if case["steps"] == 1 or n < 8:
        return [(lo, st, n)]
    a, b = n // 2, n // 4
    return [(lo, st, a), (lo + a * st, 2 * st, b), (lo + a * st + b * 2 * st, 4 * st, n - a - b)]


def _brute_shifts(case):
    """Whole-sample shifts [ndms][nchans], computed in 64 bits and rounded."""
    f32 = np.float32
    foff, tsamp = f32(-case["bw"] / case["nchans"]), float(f32(TSAMP))
    fc = float(f32(FCH1)) + float(foff) * np.arange(case["nchans"], dtype=np.float64)
    d64 = K_PLAN * (1.0 / (fc * fc) - 1.0 / (float(f32(FCH1)) * float(f32(FCH1))))
    rows = []
    for lo, st, n in _segments(case):
        dm = float(f32(lo)) + np.arange(n, dtype=np.float64) * float(f32(st))
        rows.append(np.floor(d64[None, :] * dm[:, None] / tsamp + 0.5))
    return np.concatenate(rows).astype(np.int64)


def _passes(case):
    """Subband passes: each doubles the step (and with bin0 2 the downsampling) of the one
    before and has half its calls."""
    out, lo, st, nc, b = [], 0.0, case["dmstep"], case["ncalls"], 1
    for _ in range(case["npasses"]):
        width = case["calldms"] * st
        out.append(dict(lowdm=lo, highdm=lo + nc * width, dmstep=st, sub_dmstep=width, ncalls=nc,
                        calldms=case["calldms"], ndms=nc * case["calldms"], binsize=b))
        lo, st, nc = lo + nc * width, 2 * st, max(1, nc // 2)
        if case["bin0"] == 2:
            b *= 2
    return out


def _fma32(a, b, c):
    return np.float32(np.float64(a) * np.float64(b) + np.float64(c))


def _subband_shifts(case, ps):
    """(S1 [ncalls][nchans], S2 [ncalls * calldms][nsubs]) of a pass, in the plan's 32-bit steps."""
    f32 = np.float32
    n, nsubs = case["nchans"], case["nsubs"]
    cps, tsb = n // nsubs, f32(f32(TSAMP) * f32(ps["binsize"]))
    fc = f32(FCH1) + f32(-BW / n) * np.arange(n, dtype=f32)
    dms = (K_PLAN * (1.0 / fc.astype(np.float64) / fc.astype(np.float64) -
                     1.0 / float(f32(FCH1)) / float(f32(FCH1)))).astype(f32)
    low, sub, step = f32(ps["lowdm"]), f32(ps["sub_dmstep"]), f32(ps["dmstep"])
    s1 = np.empty((ps["ncalls"], n), np.int64)
    s2 = np.empty((ps["ncalls"] * ps["calldms"], nsubs), np.int64)
    top = dms[::cps]
    half = f32(f32(ps["calldms"]) * step) / f32(2.0)
    for j in range(ps["ncalls"]):
        st = f32(_fma32(f32(j), sub, low) / tsb)
        tv = np.trunc(top * st).astype(f32)
        s1[j] = np.trunc(_fma32(dms, st, -np.repeat(tv, cps)))
        dm0 = f32(f32(low + f32(sub * f32(j))) - half)
        dm0 = dm0 if dm0 > 0 else f32(0.0)
        for k in range(ps["calldms"]):
            s2[j * ps["calldms"] + k] = np.floor(top * f32(_fma32(f32(k), step, dm0) / tsb))
    return s1, s2


# ---- inputs -------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _pulses(rng, n, nsamp, dm_hi, sigma, nchans, snr=(10.0, 40.0)):
    out = []
    for _ in range(n):
        w = int(rng.integers(1, 33))
        out.append((int(rng.integers(0, max(1, nsamp - w))), float(rng.uniform(0.0, dm_hi)), w,
                    float(rng.uniform(*snr)) * sigma / math.sqrt(nchans * w)))
    return out


def _fill_block(flat, dtype, nchans, stride, ncols, seed, bw, pulses=(), rfi=False):
    """Noise of a receiver in flat's [nchans][stride] block: 8-bit mean 128 sigma 16, 16-bit sigma
    1000, float sigma 1; dispersed boxcar pulses; with rfi, impulses of 50 sigma in 1% of the
    samples and 10-sigma sinusoids in 20 channels."""
    g, rng = _gen(seed), np.random.default_rng(seed)
    mean, sigma = {"u8": (128.0, 16.0), "i16": (0.0, 1000.0), "f32": (0.0, 1.0)}[dtype]
    view = flat[: nchans * stride].view(nchans, stride)
    fc = FCH1 - bw / nchans * np.arange(nchans)
    unit = K_PULSE * (fc ** -2 - FCH1 ** -2) / TSAMP
    if rfi:
        cols = torch.randperm(ncols, generator=g, device="cuda")[: max(1, ncols // 100)]
        tones = set(rng.choice(nchans, min(20, nchans), replace=False).tolist())
        time = torch.arange(stride, device="cuda", dtype=torch.float32)
    for c0 in range(0, nchans, 256):
        n = min(256, nchans - c0)
        v = torch.empty((n, stride), device="cuda")
        v.normal_(mean, sigma, generator=g)
        for t0, dm, w, amp in pulses:
            at = torch.from_numpy(np.floor(dm * unit[c0:c0 + n] + 0.5).astype(np.int64) + t0)
            at = (at[:, None] + torch.arange(w)[None, :]).clamp(max=ncols - 1).cuda()
            v.scatter_add_(1, at, torch.full(at.shape, float(amp), device="cuda"))
        if rfi:
            v[:, cols] += 50.0 * sigma
            for c in range(c0, c0 + n):
                if c in tones:
                    v[c - c0] += 10.0 * sigma * torch.sin(time * (6.2831853 / (8.0 + c % 180)))
        if dtype != "f32":
            info = torch.iinfo(_TORCH[dtype])
            v = v.round_().clamp_(info.min, info.max)
        view[c0:c0 + n].copy_(v)
    return view


def _series(case, seed):
    """Dedispersed series [ndms][nsamp]: noise with pulses that spread over neighbouring trials."""
    g, rng = _gen(seed), np.random.default_rng(seed)
    mean, sigma = (524288.0, 1024.0) if case["dtype"] == "i32" else (0.0, 16.0)
    ndms, nsamp = case["ndms"], case["nsamp"]
    y = torch.empty((ndms, nsamp), device="cuda")
    y.normal_(mean, sigma, generator=g)
    for _ in range(6):
        d, t, w = int(rng.integers(ndms)), int(rng.integers(nsamp)), int(rng.integers(1, 65))
        amp = float(rng.uniform(8, 20)) * sigma
        for k in range(-8, 9):
            if 0 <= d + k < ndms:
                y[d + k, t:t + w + abs(k)] += amp / math.sqrt(1.0 + abs(k)) / math.sqrt(w)
    return y.round_().to(torch.int32) if case["dtype"] == "i32" else y


def _plan(case):
    if case["kind"] == "brute":
        f = case["dtype"] == "f32"
        return m.BrutePlan(case["nchans"], FCH1, -case["bw"] / case["nchans"], TSAMP,
                           case["nsamp"], _segments(case), in_dtype=case["dtype"],
                           shift_mode="fp64_round" if f else "l1", out_dtype="f32" if f else "i32")
    return m.SubbandPlan(case["nchans"], FCH1, -BW / case["nchans"], TSAMP, case["nsamp"],
                         case["nsubs"], _passes(case), in_dtype=case["dtype"],
                         out_dtype="f32" if case["dtype"] == "f32" else "i32")


def _beams(case):
    """(nchans, nsamp, ndms, maxdm) of each beam, uneven."""
    return [(case["nchans"] * (2 if b % 3 == 1 else 1), case["nsamp"] * (1 + b % case["spread"]),
             case["ndms"] + 32 * b, case["maxdm"] * (1.0 + 0.25 * b)) for b in range(case["nbeams"])]


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed + 1)
    st = {"case": case}
    if kind in ("brute", "subband"):
        plan = _plan(case)
        info = plan.info
        ncols = info.nsamp + info.maxshift
        bw = case.get("bw", BW)
        sigma = {"u8": 16.0, "i16": 1000.0, "f32": 1.0}[case["dtype"]]
        dm_hi = float(plan.dm_values()[-1])
        st["plan"], st["in"], st["out"] = plan, plan.alloc_input(), plan.alloc_output()
        st["out"].zero_()  # (the rows of downsampled passes are filled in part)
        _fill_block(st["in"], case["dtype"], info.nchans, info.in_stride, ncols, seed, bw,
                    _pulses(rng, 4, info.nsamp, dm_hi, sigma, info.nchans))
    elif kind == "clip":
        stride = (case["nsamp"] + 15) // 16 * 16
        flat = torch.zeros(case["nchans"] * stride, dtype=_TORCH[case["dtype"]], device="cuda")
        st["fresh"] = _fill_block(flat, case["dtype"], case["nchans"], stride, case["nsamp"], seed,
                                  BW, rfi=True)
        st["block"] = torch.empty_like(st["fresh"])
    elif kind in ("boxcar", "detect"):
        st["series"] = _series(case, seed)
    elif kind == "ingest":
        st["raw"] = _raw(case, seed)
        st["stride"] = (case["nsamp"] + 15) // 16 * 16
        st["out"] = torch.zeros((case["nchans"], st["stride"]), dtype=_TORCH[case["out"]],
                                device="cuda")
    else:
        plans, fresh, d_in, d_out = [], [], [], []
        for b, (nchans, nsamp, ndms, maxdm) in enumerate(_beams(case)):
            p = m.BrutePlan(nchans, FCH1, -BW / nchans, TSAMP, nsamp, [(0.0, maxdm / ndms, ndms)],
                            in_dtype="u8", out_dtype="i32")
            i = p.info
            t = p.alloc_input()
            _fill_block(t, "u8", nchans, i.in_stride, nsamp + i.maxshift, seed + 100 * b, BW,
                        _pulses(rng, 2, nsamp, 0.9 * maxdm, 16.0, nchans))
            plans.append(p)
            fresh.append(t)
            d_in.append(t.clone())
            d_out.append(p.alloc_output())
        batch = Batch(plans)
        batch.set_buffers(d_in, d_out)
        batch.enable_clip(4.0, 4.0)
        batch.enable_detect(nwidths=9, threshold=THRESHOLD, cap=4096)
        batch.autotune()
        st.update(batch=batch, fresh=fresh, d_in=d_in, d_out=d_out)
    return st


def _raw(case, seed):
    """Raw time-major spectra as a recorder packs them."""
    g, n = _gen(seed), case["nchans"] * case["nsamp"]
    if case["nbits"] == 32:
        return torch.empty(n, device="cuda").normal_(0.0, 1.0, generator=g).view(torch.uint8)
    if case["nbits"] == 8:
        v = torch.empty(n, device="cuda").normal_(128.0, 16.0, generator=g)
        return v.round_().clamp_(0, 255).to(torch.uint8)
    return torch.randint(0, 256, (n * case["nbits"] // 8,), generator=g, device="cuda",
                         dtype=torch.uint8)


def _cands(c):
    """A candidate list's fields, in arrays of one size (zeros after the last candidate)."""
    n, out = min(len(c), SLOTS), {}
    for k in ("dm_idx", "sample", "snr", "width"):
        out[k] = np.zeros(SLOTS, c.dtype[k])
        out[k][:n] = c[k][:n]
    return out


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("brute", "subband"):
        return st["plan"].dedisperse_device(st["in"], st["out"])
    if kind == "clip":
        st["block"].copy_(st["fresh"])  # the next block arrives
        return m.rfi_clip_device(st["block"], case["nchans"], st["block"].stride(0), case["nsamp"],
                                 4.0, 4.0, dtype=case["dtype"])
    if kind == "boxcar":
        c, total = m.boxcar_detect_device(st["series"], case["nwidths"], THRESHOLD)
        return {"cands": _cands(c), "total": total}
    if kind == "detect":
        c, mean, rms, total = m.ref_detect_device(st["series"], 2.0, 0.5, THRESHOLD)
        return {"cands": _cands(c), "mean": mean, "rms": rms, "total": total}
    if kind == "ingest":
        sigproc.unpack_device(st["raw"], case["nsamp"], case["nchans"], case["nbits"], st["out"],
                              case["out"], st["stride"], invert=case["invert"])
        return st["out"]
    for a, b in zip(st["d_in"], st["fresh"]):  # the next blocks arrive
        a.copy_(b)
    st["batch"].run(graph=True)
    return {"series": list(st["d_out"]),
            "cands": [_cands(st["batch"].candidates(b)) for b in range(case["nbeams"])]}


# ---- what a pass cannot do without --------------------------------------------------------------

def _maxshift(nchans, bw, dm):
    fc = FCH1 - bw / nchans * (nchans - 1)
    return K_PLAN * (fc ** -2 - FCH1 ** -2) * dm / TSAMP


def work(case):
    kind = case["kind"]
    if kind == "brute":
        lo, st, n = _segments(case)[-1]
        e, ms = _ELEM[case["dtype"]], _maxshift(case["nchans"], case["bw"], lo + st * n)
        return {"bytes": case["nchans"] * (case["nsamp"] + ms) * e + 4.0 * case["ndms"] * case["nsamp"],
                "flops": 1.0 * case["nchans"] * case["nsamp"] * case["ndms"]}
    if kind == "subband":
        ps = _passes(case)
        ms = _maxshift(case["nchans"], BW, ps[-1]["highdm"])
        flops = out = 0.0
        for p in ps:
            ns = case["nsamp"] / p["binsize"]
            flops += ns * p["ncalls"] * (case["nchans"] + p["calldms"] * case["nsubs"])
            out += 4.0 * ns * p["ndms"]
        return {"bytes": case["nchans"] * (case["nsamp"] + ms) * _ELEM[case["dtype"]] + out,
                "flops": flops}
    if kind == "clip":  # the block's copy, then both statistics and the clipped samples
        n = case["nchans"] * case["nsamp"]
        return {"bytes": 2.0 * n * _ELEM[case["dtype"]], "flops": 6.0 * n}
    if kind == "boxcar":
        n = case["ndms"] * case["nsamp"]
        return {"bytes": 4.0 * n, "flops": 2.0 * case["nwidths"] * n}
    if kind == "detect":
        n = case["ndms"] * case["nsamp"]
        return {"bytes": 4.0 * n, "flops": 12.0 * n}
    if kind == "ingest":
        n = case["nchans"] * case["nsamp"]
        return {"bytes": n * (case["nbits"] / 8.0 + _ELEM[case["out"]]), "flops": 0.0}
    nb = fl = 0.0
    for nchans, nsamp, ndms, maxdm in _beams(case):
        nb += 2.0 * nchans * (nsamp + _maxshift(nchans, BW, maxdm)) + 4.0 * ndms * nsamp
        fl += 1.0 * nchans * nsamp * ndms
    return {"bytes": nb, "flops": fl}


# ---- results in 64 bits -------------------------------------------------------------------------

def _sum_shifted(x, shifts, nsamp):
    """out[d][t] = sum over c of x[c][t + shifts[d][c]] in 64 bits."""
    out = torch.zeros((shifts.shape[0], nsamp), dtype=torch.float64, device="cuda")
    s = torch.from_numpy(np.ascontiguousarray(shifts)).cuda()
    for c in range(x.shape[0]):
        out += x[c].unfold(0, nsamp, 1)[s[:, c]]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "brute" and case["dtype"] == "f32":
        shifts = _brute_shifts(case)
        if shifts.size * case["nsamp"] > 3e10:
            return None
        ncols = case["nsamp"] + int(shifts.max())
        stride = (ncols + 3) // 4 * 4
        x = torch.empty(case["nchans"] * stride, device="cuda")
        rng = np.random.default_rng(seed + 1)
        lo, st, n = _segments(case)[-1]
        f32 = np.float32
        dm_hi = float(f32(f32(lo) + f32(f32(n - 1) * f32(st))))
        x = _fill_block(x, "f32", case["nchans"], stride, ncols, seed, case["bw"],
                        _pulses(rng, 4, case["nsamp"], dm_hi, 1.0, case["nchans"]))
        return _sum_shifted(x.double(), shifts, case["nsamp"])
    if kind == "subband" and case["dtype"] == "f32":
        return _exact_subband(case, seed)
    if kind == "clip" and case["dtype"] == "f32":
        stride = (case["nsamp"] + 15) // 16 * 16
        flat = torch.zeros(case["nchans"] * stride, device="cuda")
        x = _fill_block(flat, "f32", case["nchans"], stride, case["nsamp"], seed, BW,
                        rfi=True).double()
        y = x[:, : case["nsamp"]]
        for dim in (1, 0):
            mu = y.mean(dim, keepdim=True)
            sig = ((y * y).mean(dim, keepdim=True) - mu * mu).clamp(min=0.0).sqrt()
            y = torch.where((y - mu).abs() >= 4.0 * sig, mu.expand_as(y), y)
        x[:, : case["nsamp"]] = y
        return x
    if kind == "detect":
        y = _series(case, seed).double()
        n = y.numel()
        mod = min(32768, n)
        k = 1
        while (k + 1) * mod < n:  # the reference's loop leaves the last chunk out
            k += 1
        z = y.reshape(-1)[: k * mod]
        mean = float(z.mean())
        rms = math.sqrt(float((z * z).mean()) - mean * mean)
        med = y.unfold(1, 5, 1).median(dim=2).values
        hit = med[(med - mean) >= rms * THRESHOLD] / rms  # (row by row: dm, then sample)
        snr = torch.zeros(SLOTS, dtype=torch.float64)
        snr[: min(len(hit), SLOTS)] = hit[:SLOTS].cpu()
        return {"cands": {"dm_idx": None, "sample": None, "snr": snr, "width": None},
                "mean": mean, "rms": rms, "total": None}
    if kind == "ingest" and case["out"] == "f32":
        x = _raw(case, seed)
        if case["nbits"] == 32:
            v = x.view(torch.float32).double()
        elif case["nbits"] == 16:
            b = x.to(torch.int64).view(-1, 2)
            v = (b[:, 0] + 256 * b[:, 1]).double()
        else:
            per = 8 // case["nbits"]
            sh = torch.arange(per, device="cuda") * case["nbits"]
            v = ((x.to(torch.int64)[:, None] >> sh) & ((1 << case["nbits"]) - 1)).reshape(-1).double()
        v = v.view(case["nsamp"], case["nchans"]).t()
        if case["invert"]:
            v = v.flip(0)
        out = torch.zeros((case["nchans"], (case["nsamp"] + 15) // 16 * 16), dtype=torch.float64,
                          device="cuda")
        out[:, : case["nsamp"]] = v
        return out
    return None  # whole numbers, or a selection among values that the search rounds itself


def _exact_subband(case, seed):
    passes = _passes(case)
    tables = [_subband_shifts(case, p) for p in passes]
    maxshift, rows, cost, dm_hi = 0, 0, 0.0, 0.0
    f32 = np.float32
    for p, (s1, s2) in zip(passes, tables):
        maxshift = max(maxshift, int(s1.max() + s2.max()) * p["binsize"])
        rows += p["ndms"]
        cost += case["nsamp"] / p["binsize"] * p["ncalls"] * (case["nchans"] + p["calldms"] * case["nsubs"])
    if cost > 3e10:
        return None
    p = passes[-1]
    half = f32(f32(p["calldms"]) * f32(p["dmstep"])) / f32(2.0)
    dm0 = f32(f32(f32(p["lowdm"]) + f32(f32(p["sub_dmstep"]) * f32(p["ncalls"] - 1))) - half)
    dm_hi = float(_fma32(f32(p["calldms"] - 1), f32(p["dmstep"]), dm0 if dm0 > 0 else f32(0.0)))
    ncols = case["nsamp"] + maxshift
    stride = (ncols + 3) // 4 * 4
    flat = torch.empty(case["nchans"] * stride, device="cuda")
    rng = np.random.default_rng(seed + 1)
    x = _fill_block(flat, "f32", case["nchans"], stride, ncols, seed, BW,
                    _pulses(rng, 4, case["nsamp"], dm_hi, 1.0, case["nchans"])).double()
    out = torch.zeros((rows, case["nsamp"]), dtype=torch.float64, device="cuda")
    row, cps = 0, case["nchans"] // case["nsubs"]
    for p, (s1, s2) in zip(passes, tables):
        b = p["binsize"]
        length, ns = ncols // b, case["nsamp"] // b
        xd = x[:, : length * b].view(case["nchans"], length, b).sum(2) if b > 1 else x[:, :length]
        n1 = ns + int(s2.max())
        z = torch.stack([_sum_shifted(xd[k * cps:(k + 1) * cps], s1[:, k * cps:(k + 1) * cps], n1)
                         for k in range(case["nsubs"])])  # [nsubs][ncalls][n1]
        for j in range(p["ncalls"]):
            n = p["calldms"]
            out[row:row + n, :ns] = _sum_shifted(z[:, j], s2[j * n:(j + 1) * n], ns)
            row += n
    return out
