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
