"""Performance cases of the correlator: what its users have it do, from a
single short dump to a full-rate sector, through the public Python binding.

A pass ends where the reference's sector loop ends (src/main.rs:2173-2683): with
the sector's dump values, i.e. the f32 spectra that go into the .cor files
(fxc.normalize) and, for the phased array, the .raw frames.  A user's program
reads the spectra back after every sector, so a pass does too; .raw frames of
sectors that are in HBM stay there, in the program's own buffer.

Kinds of cases (``kind``):
  device  one sector whose words are in HBM already (Scan.run_device)
  host    one sector from page-locked host buffers (Scan.submit / Scan.wait),
          the call that the command-line tools make for every sector
  batch   one sector each of several scans in one call (Batch.run_device_raw),
          what a multi-process schedule and the server do

Products follow the four tools: "acf" (yi-acf: both auto-spectra over the
overlap), "xcf" (yi-xcf), "corr" (yi-corr: auto- and cross-spectra), "phased"
(yi-phasedarray: phased power and re-quantised .raw frames).
"""
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path("fx-corr_b200").resolve()))
import fxc  # noqa: E402

PRODUCTS = {
    "acf": fxc.PROD_ACF | fxc.PROD_ACF_OVERLAP_ONLY,
    "xcf": fxc.PROD_XCF,
    "corr": fxc.PROD_ACF | fxc.PROD_XCF,
    "phased": fxc.PROD_PHASED | fxc.PROD_RAW,
}
OBS_HZ = 8.4e9
RHO = 0.05       # correlation of the two stations' noise
LAG = 7          # samples by which station 2's common noise lags
FFTS = (1024, 2048, 4096, 8192, 16384, 32768, 65536)


def listed():
    base = dict(kind="device", product="corr", fft=8192, nf=1, msps=512, bits1=2, bits2=2,
                shuffle="generic", lsb1=False, lsb2=False, offset_mhz=0.0, table=False, scans=1)
    return [
        # the shortest dump: under a millisecond of a 32 Msps recording, as when
        # looking for fringes in real time; latency and launches count
        dict(base, name="corr_1024_first_dump", fft=1024, nf=25, msps=32, shuffle="identity"),
        # the plain single-process run: 1 s at 32 Msps, FFT 1024, all products
        dict(base, name="corr_1024_one_second", fft=1024, nf=31250, msps=32, shuffle="identity"),
        # yi-acf on 8-bit words, an odd number of short frames
        dict(base, name="acf_2048_8bit", product="acf", fft=2048, nf=20011, bits1=8, bits2=8,
             shuffle="pairswap"),
        # yi-xcf between stations of different bit depths, a ragged last sector
        dict(base, name="xcf_4096_4bit_2bit", product="xcf", fft=4096, nf=12207, bits1=4,
             lsb1=True, offset_mhz=-8.0),
        # the full-rate scan's sector: 1 s at 1024 Msps, LSB against USB, band
        # centres 16 MHz apart, geometric table (the largest case)
        dict(base, name="corr_8192_full_rate", nf=125000, msps=1024, lsb1=True, offset_mhz=16.0,
             table=True),
        # 1-bit stations at FFT 16384 whose band shift is an odd number of bins
        dict(base, name="corr_16384_1bit_odd_shift", fft=16384, nf=8001, bits1=1, bits2=1,
             shuffle="identity", offset_mhz=2.03125),
        # the finest spectral resolution
        dict(base, name="corr_65536", fft=65536, nf=3001, lsb1=True, lsb2=True, offset_mhz=16.0),
        # yi-phasedarray: power and .raw frames at the common lengths and depths
        dict(base, name="phased_1024", product="phased", fft=1024, nf=50001, offset_mhz=4.0),
        dict(base, name="phased_8192", product="phased", nf=12503, lsb1=True, lsb2=True,
             offset_mhz=-16.0),
        dict(base, name="phased_16384_4bit", product="phased", fft=16384, nf=3001, bits1=4,
             bits2=4, offset_mhz=2.0),
        # a multi-process schedule: short sectors of scans with mixed FFT
        # lengths, bit depths and products in one call
        dict(base, name="batch_mixed_24", kind="batch", product="mixed", fft=0, nf=2**26,
             scans=24),
        # 0.1 s of the full-rate scan from host memory
        dict(base, name="host_8192", kind="host", nf=12500, msps=1024, lsb1=True,
             offset_mhz=16.0, table=True),
    ]


def draw(rng):
    """Station-samples spread over their logarithm from 2^15 to 2^30, every FFT
    length, bit depth, shuffle class, product and sideband mix."""
    kind = rng.choice(["device"] * 8 + ["host", "batch"])
    units = 2.0 ** rng.uniform(15, 30 if kind == "device" else 27)
    fft = rng.choice(FFTS)
    c = dict(kind=kind, product=rng.choice(["acf", "xcf", "corr", "corr", "phased", "phased"]),
             fft=fft, nf=max(1, int(units / (2 * fft))), msps=rng.choice([32, 256, 512, 1024]),
             bits1=rng.choice([1, 2, 2, 2, 4, 8]), bits2=0,
             shuffle=rng.choice(["identity", "pairswap", "generic", "generic"]),
             lsb1=rng.random() < 0.5, lsb2=rng.random() < 0.5, offset_mhz=0.0,
             table=rng.random() < 0.5, scans=1)
    c["bits2"] = c["bits1"] if rng.random() < 0.7 else rng.choice([1, 2, 4, 8])
    # up to an eighth of the band between the stations' centres, in whole bins
    # (any number: odd ones too); products that need no alignment have none
    c["offset_mhz"] = rng.choice([0, rng.randint(-fft // 16, fft // 16)]) * c["msps"] / fft
    if kind == "batch":
        c.update(product="mixed", fft=0, nf=int(units), scans=rng.randint(2, 24))
    return c


# ------------------------------------------------------------------- set-up

def _levels(bits):
    if bits == 1:
        return [-1.0, 1.0]
    if bits == 2:
        return [-3.0, -1.0, 1.0, 3.0]
    m = 1 << bits
    return [i - (m - 1) / 2.0 for i in range(m)]


def _gain(bits):
    """Unit-variance noise to level units: thresholds at +-0.98 sigma for 2-bit
    words, a step of about 3.5 / 2^(b-1) sigma for wider ones."""
    return 1.0 if bits == 1 else (2.0 / 0.98 if bits == 2 else (1 << (bits - 1)) / 3.5)


def _shuffle(kind, rng):
    if kind == "identity":
        return list(range(32))
    if kind == "pairswap":
        return [i ^ 1 for i in range(32)]
    p = list(range(32))
    rng.shuffle(p)
    return p


def _band(fft, fs, offset_hz):
    """compute_band_alignment (src/main.rs:360-372) for equal bandwidths, the
    centre of station 1 less that of station 2 = offset_hz."""
    v = fft // 2
    sb = int(math.floor(abs(offset_hz) / (fs / fft) + 0.5)) * (1 if offset_hz >= 0 else -1)
    a1s = max(0, -sb)
    a1e = min(v, v - sb)
    return (sb, a1s, a1e, a1s + sb)


def _scan_fields(c, seed):
    """The scan's configuration (fields of fxc.ScanConfig) and its first frame."""
    r = random.Random(seed * 1000003 + 17)
    fs = c["msps"] * 1e6
    lo = OBS_HZ + 1e6 * r.uniform(-1, 1)
    delay = dict(time_offset_s=0.0, lo1_hz=lo, lo2_hz=lo - c["offset_mhz"] * 1e6)
    table = None
    if c["table"]:
        # 1-s geometric delays (0.5 Hz fringe) with a user delay and rate
        table = 2.1e-7 + (-0.5 / OBS_HZ) * np.arange(61, dtype=np.float64)
        delay.update(delay_user_samples=0.3, extra_delay_rate_sps=0.01 / OBS_HZ,
                     clock2_delay_s=r.uniform(-4, 4) / fs, clock2_rate_sps=1e-12,
                     d_seek=math.floor(2.1e-7 * fs) / fs)
    else:
        delay.update(net_d1_base=r.uniform(-200, 200) / fs, total_rate1_base=r.uniform(-1, 1) * 2e-6,
                     total_accel1_base=1e-10, net_d2_base=r.uniform(-8, 8) / fs,
                     total_rate2_base=-3e-7)
    f = dict(fft=c["fft"], fs=fs, bits1=c["bits1"], bits2=c["bits2"], levels1=_levels(c["bits1"]),
             levels2=_levels(c["bits2"]), shuffle1=_shuffle(c["shuffle"], r),
             shuffle2=_shuffle(c["shuffle"], r), lsb1=c["lsb1"], lsb2=c["lsb2"],
             band=_band(c["fft"], fs, c["offset_mhz"] * 1e6),
             grid=0 if c["offset_mhz"] >= 0 else 1, products=PRODUCTS[c["product"]],
             w1=1.0, w2=r.choice([1.0, 0.8]), delay=delay, geom_table=table)
    return f, r.randrange(0, 1000)


def _members(c, seed):
    """The single-scan cases of a case (itself, or the scans of a batch)."""
    if c["kind"] != "batch":
        return [(c, seed)]
    r = random.Random(c["scans"] * 7919 + c["nf"])  # the schedule is the case's, not the seed's
    out = []
    for i in range(c["scans"]):
        fft = r.choice([1024, 4096, 16384])
        bits = r.choice([1, 2, 4])
        share = c["nf"] / c["scans"] * r.uniform(0.4, 1.6)
        out.append((dict(c, kind="device", product="phased" if r.random() < 1 / 3 else "corr",
                         fft=fft, nf=max(1, int(share / (2 * fft))), bits1=bits, bits2=bits,
                         lsb1=r.random() < 0.5, lsb2=r.random() < 0.5,
                         offset_mhz=2 * r.randint(-40, 40) * c["msps"] / fft,
                         shuffle=r.choice(["identity", "generic"])), seed * 64 + i))
    return out


def _raw_pair(f, nf, seed):
    """Both stations' packed words: seeded quantised Gaussian noise with a
    common component, made on the device."""
    n = nf * f["fft"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    outs = [torch.empty(n * b // 8, dtype=torch.uint8, device="cuda")
            for b in (f["bits1"], f["bits2"])]
    a, b = math.sqrt(RHO), math.sqrt(1 - RHO)
    for s0 in range(0, n, 1 << 26):
        m = min(1 << 26, n - s0)
        com = torch.randn(m + LAG, device="cuda", generator=g)
        for st in range(2):
            bits, lsb, sh = f[f"bits{st + 1}"], f[f"lsb{st + 1}"], f[f"shuffle{st + 1}"]
            x = a * (com[LAG:] if st == 0 else com[:m])
            x += b * torch.randn(m, device="cuda", generator=g)
            if lsb:
                x[1::2].neg_()
            step = 2.0 if bits <= 2 else 1.0
            code = (x * (_gain(bits) / step) + (1 << bits) / 2).floor_().clamp_(0, (1 << bits) - 1)
            code = code.to(torch.int64).view(-1, 32 // bits)
            w = (code << (torch.arange(32 // bits, device="cuda") * bits)).sum(1)
            if sh != list(range(32)):
                v = torch.zeros_like(w)
                for pos in range(32):
                    v |= ((w >> pos) & 1) << sh[pos]
                w = v
            outs[st][s0 * bits // 8:(s0 + m) * bits // 8] = w.to(torch.int32).view(torch.uint8)
    return outs


_ENGINE = []


def _engine():
    """One engine per process, as a program keeps it."""
    if not _ENGINE:
        _ENGINE.append(fxc.Engine(0))
    return _ENGINE[0]


def prepare(case, seed):
    eng = _engine()
    st = dict(kind=case["kind"], scans=[], raw1=[], raw2=[], nf=[], first=[])
    for c, s in _members(case, seed):
        f, first = _scan_fields(c, s)
        r1, r2 = _raw_pair(f, c["nf"], s)
        if case["kind"] == "host":
            r1, r2 = (torch.empty(r.numel(), dtype=torch.uint8, pin_memory=True).copy_(r).numpy()
                      for r in (r1, r2))
        for k, v in zip(("scans", "raw1", "raw2", "nf", "first"),
                        (eng.open_scan(fxc.ScanConfig(**f)), r1, r2, c["nf"], first)):
            st[k].append(v)
    if case["kind"] == "batch":
        st["batch"] = fxc.Batch(eng, use_graphs=True)
    if case["kind"] != "host":
        st["acc"] = [torch.empty(5 * s.cfg.h, dtype=torch.float64, device="cuda")
                     for s in st["scans"]]
        st["out"] = [torch.empty(n * s.cfg.bpf(s.cfg.bits_out), dtype=torch.uint8, device="cuda")
                     if s.cfg.products & fxc.PROD_RAW else None
                     for s, n in zip(st["scans"], st["nf"])]
    st["power"] = [(fxc.level_power(s.cfg.levels1), fxc.level_power(s.cfg.levels2))
                   for s in st["scans"]]
    return st


def _dumps(cfg, nf, power, r):
    """The .cor dump values of a sector (src/main.rs:2645-2683) and its .raw frames."""
    p1, p2 = power
    p12 = math.sqrt(p1 * p2)
    out = {}
    if cfg.products & fxc.PROD_ACF:
        out["acf11"] = fxc.normalize(cfg.fft, nf, p1, acc_real=r["acf11"])
        out["acf22"] = fxc.normalize(cfg.fft, nf, p2, acc_real=r["acf22"])
    if cfg.products & fxc.PROD_XCF:
        out["xcf"] = fxc.normalize(cfg.fft, nf, p12, acc_cplx=r["xcf"])
    if cfg.products & fxc.PROD_PHASED:
        out["phased"] = fxc.normalize(cfg.fft, nf, p12, acc_real=r["phased"])
    if cfg.products & fxc.PROD_RAW:
        out["raw"] = r["raw"]
    return out


def _blocks(cfg, a, raw):
    """A sector's accumulator block (5 * H doubles) by product."""
    h = cfg.h
    return dict(acf11=a[:h], acf22=a[h:2 * h], xcf=a[2 * h:4 * h].view(np.complex128),
                phased=a[4 * h:], raw=raw)


def run(st):
    scans, nf, first = st["scans"], st["nf"], st["first"]
    if st["kind"] == "host":
        r = scans[0].wait(scans[0].submit(st["raw1"][0], st["raw2"][0], nf[0], first[0]))
        return _dumps(scans[0].cfg, nf[0], st["power"][0], r)
    if st["kind"] == "device":
        scans[0].run_device(st["raw1"][0], st["raw2"][0], nf[0], first[0], st["acc"][0],
                            st["out"][0])
        scans[0].check()
        return _dumps(scans[0].cfg, nf[0], st["power"][0],
                      _blocks(scans[0].cfg, st["acc"][0].cpu().numpy(), st["out"][0]))
    st["batch"].run_device_raw(scans, st["raw1"], st["raw2"], nf, first, st["acc"], st["out"])
    acc = torch.cat(st["acc"]).cpu().numpy()  # one copy back for every accumulator
    spectra, frames, a0 = [], [], 0
    for s, n, o, p in zip(scans, nf, st["out"], st["power"]):
        d = _dumps(s.cfg, n, p, _blocks(s.cfg, acc[a0:a0 + 5 * s.cfg.h], o))
        a0 += 5 * s.cfg.h
        if "raw" in d:
            frames.append(d.pop("raw"))
        spectra += d.values()
    return {"spectra": np.concatenate(spectra), "raw": frames}


def work(case):
    """Packed words read once, dump values and .raw frames written once; nominal
    operations: two real FFTs (2.5 N log2 N each), 6.5 a sample for decode,
    rotation and accumulation, and the phased array's inverse FFT."""
    b = f = 0.0
    for c, _ in _members(case, 0):
        n, nf = c["fft"], c["nf"]
        b += nf * n * (c["bits1"] + c["bits2"]) / 8
        f += 2 * nf * n * (2.5 * math.log2(n) + 6.5)
        if c["product"] == "phased":
            b += nf * n * max(c["bits1"], c["bits2"]) / 8 + 4 * n
            f += nf * 2.5 * n * math.log2(n)
        else:
            b += {"acf": 2, "xcf": 1, "corr": 3}[c["product"]] * 4 * n
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------- in 64 bits

def _delays(f, first, nf):
    """The per-frame delay model (src/main.rs:184-241): integer shifts, fractional
    delays and carrier angles of both stations."""
    d = dict.fromkeys(("time_offset_s", "coarse_delay_s", "delay_user_samples",
                       "extra_delay_rate_sps", "clock1_delay_s", "clock1_rate_sps",
                       "clock2_delay_s", "clock2_rate_sps", "d_seek", "net_d1_base",
                       "total_rate1_base", "total_accel1_base", "net_d2_base",
                       "total_rate2_base", "total_accel2_base"), 0.0)
    d.update(f["delay"])
    fs = f["fs"]
    loc = (np.arange(first, first + nf, dtype=np.float64) + 0.5) * (f["fft"] / fs)
    t = loc + d["time_offset_s"]
    if f["geom_table"] is not None:
        tab = f["geom_table"]
        i0 = np.minimum(np.floor(loc).astype(np.int64), len(tab) - 1)
        i1 = np.minimum(i0 + 1, len(tab) - 1)
        w = np.where(i1 != i0, np.clip(loc - i0, 0.0, 1.0), 0.0)
        net = tab[i0] * (1.0 - w) + tab[i1] * w + d["coarse_delay_s"] \
            + d["delay_user_samples"] / fs + d["extra_delay_rate_sps"] * t
        c1 = d["clock1_delay_s"] + d["clock1_rate_sps"] * t
        c2 = d["clock2_delay_s"] + d["clock2_rate_sps"] * t
        full1, full2 = net + (c2 - c1), np.zeros(nf)
        tau1, tau2 = full1 - d["d_seek"], full2
    else:
        tau1 = d["net_d1_base"] + d["total_rate1_base"] * t + 0.5 * d["total_accel1_base"] * (t * t)
        tau2 = d["net_d2_base"] + d["total_rate2_base"] * t + 0.5 * d["total_accel2_base"] * (t * t)
        full1, full2 = tau1 + d["d_seek"], tau2
    out = []
    for tau, full, lo in ((tau1, full1, d["lo1_hz"]), (tau2, full2, d["lo2_hz"])):
        v = tau * fs
        i = np.copysign(np.floor(np.abs(v) + 0.5), v)
        ang = np.mod(-2 * math.pi * lo * full + math.pi, 2 * math.pi) - math.pi
        out += [torch.from_numpy(x).cuda() for x in (i, tau - i / fs, ang)]
    return out


def _decoded(raw, m, f, st):
    """m frames of a station's words as f64 samples (src/utils.rs:215-376)."""
    bits, lsb, sh = f[f"bits{st}"], f[f"lsb{st}"], f[f"shuffle{st}"]
    w = raw.view(torch.int32).to(torch.int64) & 0xFFFFFFFF
    if sh != list(range(32)):
        v = torch.zeros_like(w)
        for o in range(32):
            v |= ((w >> sh[o]) & 1) << o
        w = v
    code = (w[:, None] >> (torch.arange(32 // bits, device="cuda") * bits)) & ((1 << bits) - 1)
    x = torch.tensor(f[f"levels{st}"], dtype=torch.float64, device="cuda")[code.view(-1)]
    x = x.view(m, f["fft"])
    if lsb:
        x[:, 1::2] *= -1
    return x


def _shifted(x, s):
    """Each frame delayed by its whole number of samples, zeros shifted in."""
    n = x.shape[1]
    i = torch.arange(n, device="cuda")[None, :] - s.to(torch.int64)[:, None]
    return torch.where((i >= 0) & (i < n), torch.gather(x, 1, i.clamp(0, n - 1)), 0.0)


def _exact_one(c, seed):
    f, first = _scan_fields(c, seed)
    raws = _raw_pair(f, c["nf"], seed)
    n, nf = f["fft"], c["nf"]
    h = n // 2 + 1
    sb, a1s, a1e, a2s = f["band"]
    ov = a1e - a1s
    g0 = f["grid"] == 0
    grid = slice(a1s, a1e) if g0 else slice(a2s, a2s + ov)
    i1, f1, p1, i2, f2, p2 = _delays(f, first, nf)
    bpf = [n * f["bits1"] // 8, n * f["bits2"] // 8]
    w = -2j * math.pi * f["fs"] / n * torch.arange(h, dtype=torch.float64, device="cuda")
    acc = {k: torch.zeros(h, dtype=torch.complex128 if k == "xcf" else torch.float64,
                          device="cuda") for k in ("acf11", "acf22", "xcf", "phased")}
    step = max(1, (1 << 24) // n)
    for c0 in range(0, nf, step):
        c1 = min(nf, c0 + step)
        s = []
        for st, (fi, fr, ph) in enumerate(((i1, f1, p1), (i2, f2, p2))):
            x = _decoded(raws[st][c0 * bpf[st]:c1 * bpf[st]], c1 - c0, f, st + 1)
            z = torch.fft.rfft(_shifted(x, fi[c0:c1]), dim=1)
            z *= torch.exp(w[None, :] * fr[c0:c1, None])
            if c["product"] == "phased":  # the inverse real FFT ignores Nyquist's imaginary part
                z[:, n // 2] = z[:, n // 2].real.to(z.dtype)
            s.append(z * torch.exp(1j * ph[c0:c1, None]))
        o1, o2 = s[0][:, a1s:a1e], s[1][:, a2s:a2s + ov]
        if c["product"] == "phased":
            cb = s[0] * f["w1"] if g0 else s[1] * f["w2"]
            cb[:, grid] += o2 * f["w2"] if g0 else o1 * f["w1"]
            acc["phased"] += cb.abs().square().sum(0)
            continue
        whole = c["product"] != "acf"
        for k, z, o, mine in (("acf11", s[0], o1, g0), ("acf22", s[1], o2, not g0)):
            if mine and whole:
                acc[k] += z.abs().square().sum(0)
            else:
                acc[k][grid] += o.abs().square().sum(0)
        acc["xcf"][grid] += (o1 * o2.conj()).sum(0)
    pw = [sum(v * v for v in f[f"levels{k}"]) / len(f[f"levels{k}"]) for k in (1, 2)]
    power = dict(acf11=pw[0], acf22=pw[1], xcf=math.sqrt(pw[0] * pw[1]),
                 phased=math.sqrt(pw[0] * pw[1]))
    keep = {"acf": ("acf11", "acf22"), "xcf": ("xcf",), "corr": ("acf11", "acf22", "xcf"),
            "phased": ("phased",)}[c["product"]]
    return {k: (acc[k][:n // 2] / (0.5 * power[k] * nf * float(n) ** 2)).to(torch.complex128)
            .cpu().numpy() for k in keep}


def exact(case, seed):
    """The spectra in 64 bits; the .raw frames are bytes and have no such value."""
    parts = [_exact_one(c, s) for c, s in _members(case, seed)]
    if case["kind"] == "batch":
        return {"spectra": np.concatenate([v for p in parts for v in p.values()]),
                "raw": [None for p in parts if "phased" in p]}
    if case["product"] == "phased":
        parts[0]["raw"] = None
    return parts[0]
