"""Bins out of the band overlap hold nothing of the cross-spectrum and of the
secondary station's auto-spectrum, whatever the samples are: a level table with
infinities makes the primary's spectrum infinite or NaN everywhere, and those bins
are zero all the same.  Every correlation kernel, per scan and batched."""
import numpy as np
import pytest

import oracle
from _cases import make_scan, random_raw, to_fxc

pytestmark = pytest.mark.gpu

INF = float("inf")
DELAY = dict(net_d1_base=3.3e-8, lo1_hz=8.4e9, lo2_hz=8.4e9)


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def scan_of(fft, grid, shift, bits):
    half = fft // 2
    levels = oracle.default_levels(bits)
    levels[0], levels[-1] = -INF, INF
    band = (shift, half // 8, half - half // 8, half // 8 + shift)
    return make_scan(fft=fft, fs=512e6, bits1=bits, bits2=bits, grid=grid, band=band, delay=DELAY,
                     levels1=levels, levels2=levels)


def check(scan, got):
    _, a1s, a1e, a2s = scan.band
    start = a1s if scan.grid == 0 else a2s
    out = np.ones(scan.h, bool)
    out[start:start + a1e - a1s] = False
    secondary = got["acf22" if scan.grid == 0 else "acf11"]
    assert not np.any(secondary[out]) and not np.any(got["xcf"][out])
    assert not np.any(np.isfinite(got["xcf"][~out]))  # the infinities did arrive


# odd shifts at FFT 16384: the one-CTA pair kernel; 4-bit stations at 65536: the
# cluster kernel
@pytest.mark.parametrize("fft,shift,bits", [
    (1024, 8, 2), (2048, 0, 4), (2048, -4, 2), (4096, 8, 8), (8192, 8, 2), (16384, 8, 2),
    (16384, 3, 2), (32768, 8, 2), (65536, 16, 1), (65536, 8, 4)])
@pytest.mark.parametrize("grid", [0, 1])
def test_infinite_levels(engine, fft, shift, bits, grid):
    scan = scan_of(fft, grid, shift, bits)
    r1, r2 = random_raw(scan, 5, seed=fft + bits)
    s = engine.open_scan(to_fxc(scan))
    got = s.sector_device(dev(r1), dev(r2), 5, first_frame=1)
    s.close()
    check(scan, got)


def test_infinite_levels_batched(engine, fxc_lib):
    import torch

    scans = [scan_of(fft, k % 2, 8, 2) for k, fft in enumerate((1024, 2048, 4096, 8192, 16384))]
    raws = [random_raw(sc, 5, seed=sc.fft) for sc in scans]
    opened = [engine.open_scan(to_fxc(sc)) for sc in scans]
    acc = [torch.zeros(5 * sc.h, dtype=torch.float64, device="cuda") for sc in scans]
    batch = fxc_lib.Batch(engine)
    batch.run_device(opened, [dev(r[0]) for r in raws], [dev(r[1]) for r in raws], [5] * 5,
                     [1] * 5, acc)
    torch.cuda.synchronize()
    for sc, a in zip(scans, acc):
        a, h = a.cpu().numpy(), sc.h
        check(sc, dict(acf11=a[:h], acf22=a[h:2 * h], xcf=a[2 * h:4 * h].view(np.complex128)))
    batch.close()
    for s in opened:
        s.close()
