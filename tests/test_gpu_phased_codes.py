"""The re-quantiser of FFT 16384 forms the samples of a frame's two rows in the last
pass, keeps their codes by sample and packs them: every output width, both staging
layouts, odd samples negated or not, several frames per CTA, against the FP64 oracle.
A code may differ only where the sample lies within f32 rounding of a decision point
(1e-4 of the series' RMS, the bound of the phased parity tests)."""
import numpy as np
import pytest

import oracle
from _cases import make_scan, signal_raw, to_fxc
from test_gpu_phased import boundary_margin, dev, raw_codes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits1,bits2", [(1, 1), (2, 1), (2, 2), (1, 8), (4, 4), (8, 2), (8, 8)])
@pytest.mark.parametrize("lsb,nf", [(False, 1), (True, 310)])
def test_codes_of_two_rows(engine, bits1, bits2, lsb, nf):
    scan = make_scan(fft=16384, fs=512e6, bits1=bits1, bits2=bits2, lsb1=lsb, lsb2=lsb,
                     shuffle="generic", band=(-16, 16, 8192, 0),
                     delay=dict(net_d1_base=3.3e-7, total_rate1_base=2.1e-6, lo1_hz=8.4e9,
                                lo2_hz=8.4e9),
                     products=oracle.PROD_PHASED | oracle.PROD_RAW)
    r1, r2 = signal_raw(scan, nf, seed=bits1 + 16 * bits2, rho=0.3, delay_samples=1.4)
    s = engine.open_scan(to_fxc(scan))
    got = s.sector_device(dev(r1), dev(r2), nf, first_frame=5)
    s.close()
    x = oracle.fp64_sector_phased(scan, r1, r2, nf, first_frame=5)["series"].reshape(-1)
    g = raw_codes(got["raw"], x.size, scan.bits_out, scan.shuffle1)
    diff = g != oracle.quantise_codes(x.astype(np.float32), scan.levels1)
    assert diff.mean() < 1e-3, diff.mean()
    margin = boundary_margin(x[diff], scan.levels1)
    assert np.all(margin < 1e-4 * float(np.sqrt(np.mean(x ** 2)))), margin.max()
