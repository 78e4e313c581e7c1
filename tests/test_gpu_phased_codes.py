"""The re-quantiser takes the samples in the inverse transform's last pass, keeps their
codes by sample and packs them (FFT 16384; 4- and 8-bit output or tables without
thresholds up to FFT 8192; FFT 32768 and 65536 in a cluster), or a thread takes one index
of all rows (the four-step path): every output width, both staging layouts, odd samples
negated or not, several frames per CTA, a last iteration with frames to spare, against
the FP64 oracle.  A code may differ only where the sample lies within f32 rounding of a
decision point (1e-4 of the series' RMS, the bound of the phased parity tests)."""
import numpy as np
import pytest

import oracle
from _cases import make_scan, signal_raw, to_fxc
from test_gpu_phased import boundary_margin, dev, raw_codes

pytestmark = pytest.mark.gpu


def check(engine, scan, nf, seed):
    r1, r2 = signal_raw(scan, nf, seed=seed, rho=0.3, delay_samples=1.4)
    s = engine.open_scan(to_fxc(scan))
    got = s.sector_device(dev(r1), dev(r2), nf, first_frame=5)
    s.close()
    x = oracle.fp64_sector_phased(scan, r1, r2, nf, first_frame=5)["series"].reshape(-1)
    g = raw_codes(got["raw"], x.size, scan.bits_out, scan.shuffle1)
    diff = g != oracle.quantise_codes(x.astype(np.float32), scan.levels1)
    assert diff.mean() < 1e-3, diff.mean()
    margin = boundary_margin(x[diff], scan.levels1)
    assert np.all(margin < 1e-4 * float(np.sqrt(np.mean(x ** 2)))), margin.max()


DELAY = dict(net_d1_base=3.3e-7, total_rate1_base=2.1e-6, lo1_hz=8.4e9, lo2_hz=8.4e9)


@pytest.mark.parametrize("bits1,bits2", [(1, 1), (2, 1), (2, 2), (1, 8), (4, 4), (8, 2), (8, 8)])
@pytest.mark.parametrize("lsb,nf", [(False, 1), (True, 310)])
def test_codes_of_two_rows(engine, bits1, bits2, lsb, nf):
    scan = make_scan(fft=16384, fs=512e6, bits1=bits1, bits2=bits2, lsb1=lsb, lsb2=lsb,
                     shuffle="generic", band=(-16, 16, 8192, 0),
                     delay=DELAY, products=oracle.PROD_PHASED | oracle.PROD_RAW)
    check(engine, scan, nf, seed=bits1 + 16 * bits2)


@pytest.mark.parametrize("fft,nf", [(1024, 1), (1024, 1203), (2048, 601), (4096, 301), (8192, 301)])
@pytest.mark.parametrize("bits,down", [(4, False), (8, False), (2, True), (1, True)])
def test_codes_of_one_row(engine, fft, nf, bits, down):
    """`down`: a descending table, which has no thresholds."""
    levels = oracle.default_levels(bits)
    scan = make_scan(fft=fft, fs=512e6, bits1=bits, bits2=2, lsb1=nf > 1, lsb2=nf > 1,
                     levels1=levels[::-1] if down else levels, shuffle="generic",
                     band=(8, 0, fft // 2 - 8, 8), delay=DELAY,
                     products=oracle.PROD_PHASED | oracle.PROD_RAW)
    check(engine, scan, nf, seed=fft + bits)


@pytest.mark.parametrize("fft,nf", [(32768, 1), (32768, 81), (65536, 43)])
@pytest.mark.parametrize("bits1,bits2", [(1, 2), (2, 2)])
@pytest.mark.parametrize("grid", [0, 1])
def test_codes_of_a_clusters_rows(engine, fft, nf, bits1, bits2, grid):
    scan = make_scan(fft=fft, fs=512e6, bits1=bits1, bits2=bits2, lsb1=nf > 1, lsb2=nf > 1,
                     grid=grid, shuffle="generic", band=(-64, 64, fft // 2, 0), delay=DELAY,
                     products=oracle.PROD_PHASED | oracle.PROD_RAW)
    check(engine, scan, nf, seed=fft + bits1 + grid)


@pytest.mark.parametrize("fft,shift", [(32768, 3), (65536, 16)])
@pytest.mark.parametrize("bits1,bits2", [(1, 4), (2, 4), (4, 4), (8, 1)])
@pytest.mark.parametrize("nf", [1, 67])
def test_codes_of_all_rows(engine, fft, shift, bits1, bits2, nf):
    scan = make_scan(fft=fft, fs=512e6, bits1=bits1, bits2=bits2, lsb1=nf > 1, lsb2=nf > 1,
                     shuffle="generic", band=(shift, 0, fft // 2 - shift, shift), delay=DELAY,
                     products=oracle.PROD_PHASED | oracle.PROD_RAW)
    check(engine, scan, nf, seed=fft + bits1)
