"""The reductions of the per-CTA partials at the edges of their two forms: one
slot, the last count of the narrow form (63), the first of the wide one (64),
a ragged share per warp and every slot of a full grid, against the FP64
oracle with the tolerance of _cases.py."""
import numpy as np
import pytest

import oracle
from _cases import assert_sector_close, assert_spectra_close, make_scan, signal_raw, to_fxc

pytestmark = pytest.mark.gpu


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


DELAY = dict(net_d1_base=3.3e-7, total_rate1_base=2.1e-6, lo1_hz=8.4e9, lo2_hz=8.4e9)


# FFT 4096 runs one frame pair per CTA iteration, two CTAs per SM: nf slots up to 296
@pytest.mark.parametrize("nf", [1, 63, 64, 65, 297])
@pytest.mark.parametrize("products", [oracle.PROD_ACF | oracle.PROD_XCF,
                                      oracle.PROD_PHASED | oracle.PROD_RAW])
def test_partials_reduction_edges(engine, nf, products):
    scan = make_scan(fft=4096, fs=512e6, band=(40, 0, 2008, 40), delay=DELAY, products=products)
    r1, r2 = signal_raw(scan, nf, seed=nf + 17, rho=0.3, delay_samples=2.6)
    s = engine.open_scan(to_fxc(scan))
    got = s.sector_device(dev(r1), dev(r2), nf, first_frame=5)
    s.close()
    if products & oracle.PROD_ACF:
        ref = oracle.fp64_sector_corr(scan, r1, r2, nf, first_frame=5)
        assert_sector_close(got, ref, scan, f"nf={nf}", nf=nf)
        assert np.all(got["phased"] == 0)
    else:
        ref = oracle.fp64_sector_phased(scan, r1, r2, nf, first_frame=5)
        assert_spectra_close(got["phased"], ref["phased"], f"phased power nf={nf}")
        assert np.all(got["acf11"] == 0) and np.all(got["xcf"] == 0)
