"""The FFT 1024..4096 correlation kernel against the FP64 oracle where its decode
and accumulation change form: integer shifts at the edges of the half of a frame
that is decoded unchecked, every bit depth and shuffle class, both grids, band
shifts of either sign, none, and overlaps that end inside a warp's bins, frame
counts that do not fill a CTA iteration, each product subset.  Tolerance of
_cases.py."""
import numpy as np
import pytest

import oracle
from _cases import assert_sector_close, make_scan, signal_raw, to_fxc

pytestmark = pytest.mark.gpu

CORR = oracle.PROD_ACF | oracle.PROD_XCF


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def check(engine, scan, nf, seed, what):
    r1, r2 = signal_raw(scan, nf, seed=seed, rho=0.3, delay_samples=2.6)
    s = engine.open_scan(to_fxc(scan))
    got = s.sector_device(dev(r1), dev(r2), nf, first_frame=3)
    s.close()
    ref = oracle.fp64_sector_corr(scan, r1, r2, nf, first_frame=3)
    full = oracle.fp64_sector_corr(
        __import__("dataclasses").replace(scan, products=CORR), r1, r2, nf, first_frame=3)
    assert_sector_close(got, ref, scan, what, nf=nf, ref_acf=full)
    if not scan.products & oracle.PROD_ACF:
        assert not np.any(got["acf11"]) and not np.any(got["acf22"])
    if not scan.products & oracle.PROD_XCF:
        assert not np.any(got["xcf"])


def delays(fs, s1, s2):
    return dict(net_d1_base=s1 / fs + 0.2 / fs, net_d2_base=s2 / fs - 0.1 / fs,
                lo1_hz=8.4e9, lo2_hz=8.4e9)


@pytest.mark.parametrize("fft", [1024, 2048, 4096])
@pytest.mark.parametrize("edge", [0, 1, 511, 512, 513, 1023, 1025])
def test_shift_edges(engine, fft, edge):
    # in 1024ths of a frame: 512 is half a frame, 8 N/16 samples
    s = edge * (fft // 1024) + (edge % 2) * (fft // 1024 - 1)
    fs = 512e6
    for s1, s2 in ((s, -s), (-s, s)):
        scan = make_scan(fft=fft, fs=fs, delay=delays(fs, s1, s2), shuffle="generic", lsb1=True)
        check(engine, scan, 9, fft + edge, f"shifts {s1} {s2}")


@pytest.mark.parametrize("fft", [1024, 2048, 4096])
@pytest.mark.parametrize("bits1,bits2,shuffle", [
    (1, 1, "generic"), (1, 2, "identity"), (2, 2, "pairswap"), (2, 2, "sample2"),
    (2, 2, "generic"), (4, 2, "generic"), (4, 4, "identity"), (8, 8, "generic"),
    (8, 1, "pairswap")])
def test_depths_and_shuffles(engine, fft, bits1, bits2, shuffle):
    fs = 512e6
    for lsb in ((False, False), (True, False), (True, True)):
        scan = make_scan(fft=fft, fs=fs, bits1=bits1, bits2=bits2, shuffle=shuffle,
                         lsb1=lsb[0], lsb2=lsb[1], delay=delays(fs, 37, -5),
                         band=(3, 0, fft // 2 - 7, 3))
        check(engine, scan, 7, fft + 10 * bits1 + bits2, f"{bits1}/{bits2} {shuffle} {lsb}")


@pytest.mark.parametrize("fft", [1024, 2048, 4096])
@pytest.mark.parametrize("grid", [0, 1])
@pytest.mark.parametrize("products", [CORR, oracle.PROD_XCF, oracle.PROD_ACF,
                                      oracle.PROD_ACF | oracle.PROD_ACF_OVERLAP_ONLY])
def test_bands_and_products(engine, fft, grid, products):
    h = fft // 2
    fs = 512e6
    # no shift over every bin; either sign; an odd shift; an overlap of one bin; one
    # that ends inside a warp
    for band in ((0, 0, h + 1, 0), (5, 0, h - 5, 5), (-7, 7, h, 0), (h // 2, 0, h // 2 + 1, h // 2),
                 (0, 17, 18, 17), (-3, 100, 133, 97)):
        scan = make_scan(fft=fft, fs=fs, grid=grid, band=band, products=products,
                         delay=delays(fs, 11, 4))
        check(engine, scan, 10, fft + grid, f"grid {grid} band {band} products {products}")


@pytest.mark.parametrize("fft", [1024, 2048, 4096])
@pytest.mark.parametrize("grid", [0, 1])
@pytest.mark.parametrize("bits1,bits2,shuffle", [
    (1, 4, "generic"), (2, 8, "pairswap"), (4, 2, "sample2"), (8, 4, "generic"),
    (4, 8, "identity"), (2, 2, "generic")])
def test_decode_bit_exact(engine, fft, grid, bits1, bits2, shuffle):
    """The kernels' own decode, through the decode stage: rewritten words and raw ones,
    integer shifts of every size, whichever station is the primary; frame counts that
    leave a CTA iteration half empty."""
    fs, nf = 32e6, 39
    delay = dict(net_d1_base=-1.3 * fft / fs, total_rate1_base=2.7 / 40, net_d2_base=5.0 / fs,
                 total_rate2_base=-0.05)
    scan = make_scan(fft=fft, fs=fs, bits1=bits1, bits2=bits2, shuffle=shuffle, lsb1=True, grid=grid,
                     delay=delay, seed=fft + bits1)
    rng = np.random.Generator(np.random.PCG64(fft + bits2))
    raws = [rng.integers(0, 256, nf * scan.bpf(b), dtype=np.uint8) for b in (bits1, bits2)]
    s = engine.open_scan(to_fxc(scan))
    got = s.decode(dev(raws[0]), dev(raws[1]), nf, first_frame=3)
    s.check()
    ents = oracle.c_delay_entries(scan, 3, nf)
    for x, raw, bits, sh, lv, lsb, key in zip(
            got, raws, (bits1, bits2), (scan.shuffle1, scan.shuffle2),
            (scan.levels1, scan.levels2), (True, False), ("int1", "int2")):
        x, bpf = x.cpu().numpy(), scan.bpf(bits)
        for i in range(nf):
            e = oracle.c_decode(raw[i * bpf:(i + 1) * bpf], fft, bits, sh, lv, lsb)
            np.testing.assert_array_equal(x[i], oracle.c_shift(e, ents[key][i]))
    assert min(ents["int1"]) <= -fft and max(ents["int1"]) >= fft
    s.close()


@pytest.mark.parametrize("fft,fpc", [(1024, 1), (1024, 2), (1024, 4), (2048, 1), (2048, 2),
                                     (2048, 4), (4096, 1), (4096, 2)])
def test_many_iterations(engine, fxc_lib, fft, fpc):
    """CTAs with dozens of iterations (a batch's items of 96 frames and of the 13 left):
    buffers that take turns, two copies in flight while words are rewritten in place,
    several flushes and a ragged last run."""
    import torch

    nf, fs, half = 109, 512e6, fft // 2
    scans = []
    for k, (bits, shuffle, grid, band) in enumerate([
            (4, "generic", 0, (0, 0, half + 1, 0)), (8, "generic", 1, (-7, 7, half, 0)),
            (2, "generic", 0, (5, 100, half - 90, 105)), (1, "identity", 1, (0, 33, half, 33)),
            (8, "pairswap", 0, (3, 0, half - 7, 3))]):
        scan = make_scan(fft=fft, fs=fs, bits1=bits, bits2=bits, shuffle=shuffle, grid=grid, band=band,
                         lsb1=k % 2 == 0, delay=delays(fs, 11 + 40 * k, 4 - 9 * k), seed=k)
        scans.append((scan, *signal_raw(scan, nf, seed=fft + k, rho=0.3, delay_samples=2.6)))
    opened = [engine.open_scan(to_fxc(sc)) for sc, *_ in scans]
    acc = [torch.zeros(5 * (half + 1), dtype=torch.float64, device="cuda") for _ in scans]
    batch = fxc_lib.Batch(engine)
    batch.set_shape(fft, fpc, 96)
    batch.run_device(opened, [dev(r1) for _, r1, _ in scans], [dev(r2) for *_, r2 in scans],
                     [nf] * len(scans), [3] * len(scans), acc)
    torch.cuda.synchronize()
    for (sc, r1, r2), s, a in zip(scans, opened, acc):
        s.check()
        a, h = a.cpu().numpy(), half + 1
        got = dict(acf11=a[:h], acf22=a[h:2 * h], xcf=a[2 * h:4 * h].view(np.complex128))
        ref = oracle.fp64_sector_corr(sc, r1, r2, nf, first_frame=3)
        assert_sector_close(got, ref, sc, f"{fft} {fpc} {sc.bits1} bits", nf=nf, ref_acf=ref)
        s.close()
    batch.close()
