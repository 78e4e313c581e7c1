"""The phased re-quantiser's decision thresholds against the nearest-level
search.  A descending level table takes the search, an ascending one (where it
qualifies) the thresholds; with the levels reversed and station 1's input codes
complemented the samples are the same bit for bit, so the output codes are each
other's complements except where a sample ties between two levels, which the
first index wins: within an ulp of a decision point, about 1e-7 of the samples.
Every kernel that re-quantises (N <= 8192 with and without votes, the two-row
kernel's layouts, the cluster kernel, the four-step path), 1 to 8 bits, uniform
and uneven tables."""
import dataclasses

import numpy as np
import pytest

import oracle
from _cases import make_scan, signal_raw, to_fxc

pytestmark = pytest.mark.gpu

UNEVEN2 = [-3.3359, -1.0, 1.2, 4.1]
UNEVEN4 = [float(np.sign(i - 7.5) * abs(i - 7.5) ** 1.3) for i in range(16)]
PROD = oracle.PROD_PHASED | oracle.PROD_RAW
DELAY = dict(net_d1_base=3.3e-7, lo1_hz=8.4e9, lo2_hz=8.4e9)


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def phased_raw(engine, scan, r1, r2, nf):
    s = engine.open_scan(to_fxc(scan))
    raw = s.sector_device(dev(r1), dev(r2), nf, first_frame=1)["raw"]
    s.close()
    return raw


@pytest.mark.parametrize("fft,bits,levels,lsb", [
    (1024, 2, None, True), (1024, 1, None, False), (2048, 2, UNEVEN2, False),
    (4096, 2, UNEVEN2, True), (4096, 4, None, False), (4096, 8, None, True),
    (8192, 2, None, False), (8192, 4, UNEVEN4, True), (16384, 2, UNEVEN2, True),
    (16384, 1, None, False), (16384, 4, None, True), (16384, 8, None, False),
    (32768, 2, None, True), (65536, 4, None, False)])
def test_thresholds_equal_search(engine, fft, bits, levels, lsb):
    up = list(levels) if levels else oracle.default_levels(bits)
    nf = max(9, 200_000 // fft)
    scan = make_scan(fft=fft, fs=512e6, bits1=bits, bits2=bits, levels1=up, delay=DELAY,
                     products=PROD, lsb1=lsb, lsb2=lsb, shuffle="generic",
                     band=(8, 0, fft // 2 - 8, 8))
    r1, r2 = signal_raw(scan, nf, seed=fft + bits, rho=0.4)
    down = dataclasses.replace(scan, levels1=up[::-1])
    a = phased_raw(engine, scan, r1, r2, nf)
    b = phased_raw(engine, down, r1 ^ np.uint8(255), r2, nf)
    differ = int(np.count_nonzero(a != (b ^ np.uint8(255))))
    assert differ <= 3, (differ, a.size)
    assert len(np.unique(a)) > 1


@pytest.mark.parametrize("fft,bits", [(1024, 2), (4096, 1), (8192, 4), (16384, 2), (16384, 4)])
def test_far_beyond_the_levels_all_tie(engine, fft, bits):
    """So far out that every rounded distance is the same: the first level."""
    scan = make_scan(fft=fft, fs=512e6, bits1=bits, bits2=bits, delay=DELAY, products=PROD,
                     w1=1e30, w2=1e30)
    r1, r2 = signal_raw(scan, 9, seed=fft, rho=0.4)
    assert not np.any(phased_raw(engine, scan, r1, r2, 9))


@pytest.mark.parametrize("fft,bits", [
    (1024, 2), (8192, 2), (2048, 4), (4096, 8), (16384, 2), (16384, 4), (16384, 8), (32768, 2),
    (32768, 4), (65536, 2), (65536, 8)])
def test_tables_in_any_order(engine, fft, bits):
    """Levels in no order (sign and magnitude, two's complement) take the search, four
    samples at a time: with station 1's codes renumbered the same way the samples are
    the same, and so are the output's but for their numbers and ties."""
    rng = np.random.Generator(np.random.PCG64(fft + bits))
    up, nf = oracle.default_levels(bits), max(9, 200_000 // fft)
    number = rng.permutation(1 << bits)  # new number of the old code
    renumbered = [0.0] * (1 << bits)
    for old, new in enumerate(number):
        renumbered[new] = up[old]
    byte = np.zeros(256, np.uint8)
    for v in range(256):
        for s in range(0, 8, bits):
            byte[v] |= number[(v >> s) & ((1 << bits) - 1)] << s
    scan = make_scan(fft=fft, fs=512e6, bits1=bits, bits2=bits, levels1=up, delay=DELAY,
                     products=PROD, lsb1=True, lsb2=True, band=(8, 0, fft // 2 - 8, 8))
    r1, r2 = signal_raw(scan, nf, seed=fft + bits, rho=0.4)
    a = phased_raw(engine, scan, r1, r2, nf)
    b = phased_raw(engine, dataclasses.replace(scan, levels1=renumbered), byte[r1], r2, nf)
    differ = int(np.count_nonzero(byte[a] != b))
    assert differ <= 3, (differ, a.size)
    assert len(np.unique(a)) > 1
