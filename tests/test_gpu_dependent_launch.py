"""The kernels of a sector call overlap their set-up with their predecessor's end.
Sector calls queued back to back on one stream, with two scans taking turns and
no synchronisation between them, and a call captured in a CUDA graph and replayed,
give what each call gives alone, bit for bit, for every kernel of the path."""
import numpy as np
import pytest

import oracle
from _cases import make_scan, signal_raw, to_fxc

pytestmark = pytest.mark.gpu

CORR = oracle.PROD_ACF | oracle.PROD_XCF
PHASED = oracle.PROD_PHASED | oracle.PROD_RAW
CASES = [(1024, 0, CORR), (4096, 3, CORR), (8192, 16, CORR), (16384, 4, CORR), (16384, 5, CORR),
         (65536, 8, CORR), (65536, 5, CORR), (1024, 3, PHASED), (8192, 4, PHASED),
         (16384, 4, PHASED), (65536, 8, PHASED), (32768, 5, PHASED), (2048, 2, CORR | PHASED)]


@pytest.mark.parametrize("fft,shift,products", CASES)
def test_back_to_back_and_captured(engine, fft, shift, products):
    import torch

    jobs = []
    for k, nf in enumerate((3, 301)):
        sc = make_scan(fft=fft, fs=512e6, band=(shift, 0, fft // 2 - shift, shift),
                       products=products, shuffle="generic", seed=k,
                       delay=dict(net_d1_base=(3 + k) * 1e-8, total_rate1_base=2e-6,
                                  lo1_hz=8.4e9, lo2_hz=8.4e9))
        nf = min(nf, 2_000_000 // fft + 2)
        r1, r2 = (torch.from_numpy(np.ascontiguousarray(r)).cuda()
                  for r in signal_raw(sc, nf, seed=fft + k, rho=0.3))
        s = engine.open_scan(to_fxc(sc))
        raw = (torch.zeros(nf * s.cfg.bpf(s.cfg.bits_out), dtype=torch.uint8, device="cuda")
               if products & oracle.PROD_RAW else None)
        acc = torch.full((5 * s.cfg.h,), 7.0, dtype=torch.float64, device="cuda")
        jobs.append((s, r1, r2, nf, acc, raw))

    def call(j, first, acc):
        s, r1, r2, nf, _, raw = j
        s.run_device(r1, r2, nf, first, acc, raw)

    alone = []
    for j in jobs:
        per = []
        for first in (0, 40):
            call(j, first, j[4])
            torch.cuda.synchronize()
            per.append((j[4].clone(), None if j[5] is None else j[5].clone()))
            j[4].fill_(7.0)
        alone.append(per)
        j[0].check()

    outs = []
    for rep in range(4):  # scans and first frames take turns, nothing waits
        for k, j in enumerate(jobs):
            for i, first in enumerate((0, 40)):
                acc = torch.full_like(j[4], 7.0)
                call(j, first, acc)
                outs.append((k, i, acc, None if j[5] is None else j[5].clone()))
    torch.cuda.synchronize()
    for k, i, acc, raw in outs:
        assert torch.equal(acc, alone[k][i][0])
        if raw is not None:
            assert torch.equal(raw, alone[k][i][1])

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for j in jobs:
            call(j, 40, j[4])
    for j in jobs:
        j[4].fill_(7.0)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    for k, j in enumerate(jobs):
        assert torch.equal(j[4], alone[k][1][0])
        j[0].check()
        j[0].close()
