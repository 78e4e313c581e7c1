"""Shuffles that move whole samples (fields may change places, every field's bits in
one common order) are decoded without rewriting the words; one that tears a single
sample apart is not.  The same samples under such a shuffle and under the identity
give the same spectra and .raw codes, bit for bit, in every kernel and bit depth."""
import dataclasses

import numpy as np
import pytest

import oracle
from _cases import make_scan, random_raw, to_fxc

pytestmark = pytest.mark.gpu

CORR = oracle.PROD_ACF | oracle.PROD_XCF
PHASED = oracle.PROD_PHASED | oracle.PROD_RAW


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def whole_shuffle(bits, kind, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    order = np.arange(bits) if kind == "fields" else rng.permutation(bits)
    if kind == "pairswap":
        return [i ^ 1 for i in range(32)]
    fields = rng.permutation(32 // bits)
    sh = [int(fields[o // bits]) * bits + int(order[o % bits]) for o in range(32)]
    if kind == "torn":
        a, b = 0, 32 - bits  # a bit of the first sample against one of the last
        sh[a], sh[b] = sh[b], sh[a]
    return sh


def shuffled(raw, sh):
    w = raw.view("<u4")
    out = np.zeros_like(w)
    for o in range(32):
        out |= ((w >> np.uint32(o)) & np.uint32(1)) << np.uint32(sh[o])
    return out.view(np.uint8)


def run(engine, scan, r1, r2, nf):
    s = engine.open_scan(to_fxc(scan))
    got = s.sector_device(dev(r1), dev(r2), nf, first_frame=2)
    s.close()
    return got


@pytest.mark.parametrize("fft", [1024, 4096, 8192, 16384, 32768, 65536])
@pytest.mark.parametrize("bits", [2, 4, 8])
@pytest.mark.parametrize("kind", ["pairswap", "fields", "both", "torn"])
def test_same_samples_same_products(engine, fft, bits, kind):
    nf = max(2, 40_000 // fft)
    for products, shift in ((CORR, 8), (CORR, 3), (PHASED, 8)):
        scan = make_scan(fft=fft, fs=512e6, bits1=bits, bits2=bits, lsb1=True, products=products,
                         band=(shift, 0, fft // 2 - shift, shift),
                         delay=dict(net_d1_base=2e-8, lo1_hz=8.4e9, lo2_hz=8.4e9))
        r1, r2 = random_raw(scan, nf, seed=fft + bits)
        ref = run(engine, scan, r1, r2, nf)
        sh1, sh2 = whole_shuffle(bits, kind, fft), whole_shuffle(bits, kind, fft + 1)
        got = run(engine, dataclasses.replace(scan, shuffle1=sh1, shuffle2=sh2),
                  shuffled(r1, sh1), shuffled(r2, sh2), nf)
        for k in ("acf11", "acf22", "xcf", "phased"):
            assert np.array_equal(got[k], ref[k]), (products, shift, k)
        if products == PHASED:  # ant1's shuffle applied to the output words
            assert np.array_equal(got["raw"], shuffled(ref["raw"], sh1))


@pytest.mark.parametrize("bits", [2, 4, 8])
@pytest.mark.parametrize("kind", ["pairswap", "fields", "both", "torn"])
def test_same_samples_same_products_2048(engine, bits, kind):
    test_same_samples_same_products(engine, 2048, bits, kind)
