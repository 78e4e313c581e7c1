"""Work items of short sectors in a batch: sector lengths at the edges of the
item rule (one frame, fewer frames than items, a ragged last item, frames that
do not fill a CTA iteration) for each group, all groups side by side in one
call, against the per-scan path: .raw bytes equal, spectra within the FP32
tolerance of _cases.py; the same bit for bit with and without graphs."""
import numpy as np
import pytest

import oracle
from _cases import assert_sector_close, assert_spectra_close, make_scan, signal_raw, to_fxc

pytestmark = pytest.mark.gpu

DELAY = dict(net_d1_base=3.3e-7, total_rate1_base=2.1e-6, lo1_hz=8.4e9, lo2_hz=8.4e9)
CORR = oracle.PROD_ACF | oracle.PROD_XCF
PHASED = oracle.PROD_PHASED | oracle.PROD_RAW


@pytest.mark.parametrize("scale", [0, 1, 2])
def test_short_sector_items(engine, fxc_lib, scale):
    import torch

    # the least item of FFT n is 32768 / n frames: nf below it, one more than
    # 24 (32) items of it, and a ragged multiple
    def length(n, parts):
        lo = 32768 // n
        return (1, parts * lo + 1, 3 * parts * lo - 5)[scale]

    items = []
    for k, (n, prod) in enumerate([(n, p) for n in (1024, 2048, 4096, 8192, 16384)
                                   for p in (CORR, PHASED)]):
        nf = length(n, 24 if prod == CORR else 32)
        nf = min(nf, 4_000_000 // n)
        sc = make_scan(fft=n, fs=512e6, band=(8, 0, n // 2 - 16, 8), delay=DELAY, products=prod,
                       shuffle="generic", seed=k)
        r1, r2 = signal_raw(sc, nf, seed=100 * scale + k, rho=0.3, delay_samples=2.6)
        d1, d2 = (torch.from_numpy(np.ascontiguousarray(r)).cuda() for r in (r1, r2))
        items.append((sc, engine.open_scan(to_fxc(sc)), d1, d2, nf))

    def run(batch):
        acc = [torch.zeros(5 * s.cfg.h, dtype=torch.float64, device="cuda")
               for _, s, *_ in items]
        raw = [torch.zeros(nf * s.cfg.bpf(s.cfg.bits_out), dtype=torch.uint8, device="cuda")
               if sc.products == PHASED else None for sc, s, _, _, nf in items]
        batch.run_device_raw([i[1] for i in items], [i[2] for i in items],
                             [i[3] for i in items], [i[4] for i in items], [3] * len(items),
                             acc, raw)
        torch.cuda.synchronize()
        return [a.cpu().numpy() for a in acc], [None if r is None else r.cpu().numpy() for r in raw]

    acc, raw = run(fxc_lib.Batch(engine))
    acc_g, raw_g = run(fxc_lib.Batch(engine, use_graphs=True))
    for (sc, s, d1, d2, nf), a, ag, r, rg in zip(items, acc, acc_g, raw, raw_g):
        assert np.array_equal(a, ag)
        one = s.sector_device(d1, d2, nf, first_frame=3)
        h = sc.fft // 2 + 1
        if sc.products == PHASED:
            assert np.array_equal(r, rg) and np.array_equal(r, one["raw"])
            assert_spectra_close(a[4 * h:], one["phased"], f"fft {sc.fft} nf {nf}")
        else:
            got = dict(acf11=a[:h], acf22=a[h:2 * h], xcf=a[2 * h:4 * h].view(np.complex128))
            assert_sector_close(got, one, sc, f"fft {sc.fft} nf {nf}", nf=nf)
        s.close()


@pytest.mark.parametrize("fft,nf,many", [(1024, 70, 2070), (2048, 100, 1182), (4096, 75, 591),
                                         (8192, 33, 294), (8192, 101, 294), (16384, 21, 147),
                                         (1024, 300, 891), (2048, 130, 900), (4096, 150, 350)])
def test_short_sector_alone_and_among_many(engine, fxc_lib, fft, nf, many):
    """A short sector runs in parts where it is alone and whole among many (so many that
    they fill the CTAs of 148 SMs evenly), or, where they do not, in items of several
    runs: the same sums bit for bit, ragged last run included."""
    import torch

    scans = []
    for k, (grid, shuffle, bits) in enumerate([(0, "generic", 2), (1, "identity", 2),
                                               (0, "generic", 4)]):
        sc = make_scan(fft=fft, fs=512e6, bits1=bits, bits2=2, grid=grid, shuffle=shuffle,
                       band=(-8, 40, fft // 2, 32), delay=DELAY, seed=k)
        r1, r2 = signal_raw(sc, nf, seed=fft + k, rho=0.3, delay_samples=2.6)
        scans.append((sc, *(torch.from_numpy(np.ascontiguousarray(r)).cuda() for r in (r1, r2))))
    opened = [[engine.open_scan(to_fxc(sc)) for sc, *_ in scans]
              for _ in range(-(-many // len(scans)))]

    def run(copies, graphs):
        acc = [[torch.zeros(5 * (fft // 2 + 1), dtype=torch.float64, device="cuda")
                for _ in scans] for _ in copies]
        n = len(copies) * len(scans)
        batch = fxc_lib.Batch(engine, use_graphs=graphs)
        batch.run_device([s for c in copies for s in c], [d1 for _ in copies for _, d1, _ in scans],
                         [d2 for _ in copies for _, _, d2 in scans], [nf] * n, [3] * n,
                         [a for c in acc for a in c])
        torch.cuda.synchronize()
        batch.close()
        return acc

    alone, among = run(opened[:1], False)[0], run(opened, False) + run(opened, True)
    for k, (sc, d1, d2) in enumerate(scans):
        for c in among:
            assert torch.equal(c[k], alone[k])
        one = opened[0][k].sector_device(d1, d2, nf, first_frame=3)
        a, h = alone[k].cpu().numpy(), fft // 2 + 1
        got = dict(acf11=a[:h], acf22=a[h:2 * h], xcf=a[2 * h:4 * h].view(np.complex128))
        assert_sector_close(got, one, sc, f"fft {fft} nf {nf}", nf=nf)
    for c in opened:
        for s in c:
            s.close()


def test_little_budget(engine, fxc_lib):
    """An engine whose budget has room for its scans and half of a call's partials: the
    call is taken, with the same sums bit for bit."""
    import torch

    sc = make_scan(fft=1024, fs=512e6, band=(-8, 40, 512, 32), delay=DELAY, shuffle="generic")
    nf, n = 300, 24  # ten items, 10 x 16416 bytes of partials, a sector
    r1, r2 = signal_raw(sc, nf, seed=5, rho=0.3, delay_samples=2.6)
    d1, d2 = (torch.from_numpy(np.ascontiguousarray(r)).cuda() for r in (r1, r2))

    def run(eng, scans):
        acc = [torch.zeros(5 * 513, dtype=torch.float64, device="cuda") for _ in range(n)]
        batch = fxc_lib.Batch(eng)
        batch.run_device(scans, [d1] * n, [d2] * n, [nf] * n, [3 + k for k in range(n)], acc)
        torch.cuda.synchronize()
        batch.close()
        return acc

    def opened(budget):
        eng = fxc_lib.Engine(0, hbm_budget_bytes=budget)
        try:
            return eng, [eng.open_scan(to_fxc(sc)) for _ in range(n)]
        except fxc_lib.FxcError as e:
            assert e.status == fxc_lib.EBUSY
            eng.close()
            return None

    lo, hi = 1 << 20, 1 << 30  # too little for the scans, enough
    while hi - lo > 1 << 18:
        mid = (lo + hi) // 2
        got = opened(mid)
        lo, hi = (lo, mid) if got else (mid, hi)
        if got:
            got[0].close()
    eng, scans = opened(hi + n * 10 * 16416 // 2)
    ref_scans = [engine.open_scan(to_fxc(sc)) for _ in range(n)]
    for a, b in zip(run(eng, scans), run(engine, ref_scans)):
        assert torch.equal(a, b)
    eng.close()
    for s in ref_scans:
        s.close()
