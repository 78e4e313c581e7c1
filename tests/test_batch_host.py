"""The host side of the batched sectors (batch.cu) on the CPU: the file is linked
with a fake of the CUDA runtime (fake_cudart.cpp) and driven by
batch_host_check.cu, which logs every launch with the launches before it and the
work items of its group."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
OK, EBUSY = 0, -6


@pytest.fixture(scope="module")
def batch(tmp_path_factory):
    """batch(command, *sectors, budget, fail_at) -> parsed output of the driver."""
    from fxc import build

    tmp = tmp_path_factory.mktemp("batch_host")
    inc = ["-I", str(ROOT / "include"), "-I", str(ROOT / "fx-corr_b200" / "csrc"),
           "-I", str(ROOT / "tests")]
    cxx = shutil.which("g++") or "g++"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", str(Path(build.nvcc()).parents[1] / "include"),
                    "-c", str(ROOT / "tests" / "fake_cudart.cpp"), "-o", str(tmp / "fake.o")],
                   check=True)
    subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1",
                    "-cudart", "none", "--diag-suppress", "128", *inc,
                    str(ROOT / "fx-corr_b200" / "csrc" / "batch.cu"),
                    str(ROOT / "tests" / "batch_host_check.cu"), str(tmp / "fake.o"),
                    "-o", str(tmp / "check")], check=True)

    def call(command, *sectors, budget=0, fail_at=-1):
        r = subprocess.run([str(tmp / "check"), command, str(budget), str(fail_at),
                            *[":".join(map(str, s)) for s in sectors]],
                           capture_output=True, text=True, check=True)
        out = dict(launches=[])
        for line in r.stdout.splitlines():
            w = line.split()
            if w[0] == "item":
                out["launches"][-1]["items"].append(tuple(map(int, w[1:])))
            elif w[0].isdigit():
                out["launches"].append(dict(name=w[1], group=int(w[2]),
                                            before=set(map(int, w[4:])), items=[]))
            elif w[0] == "stream":
                out["stream"] = set(map(int, w[1:]))
            else:
                out[w[0]] = int(w[1])
        assert out["left"] == 0  # every reserved byte was given back
        return out

    return call


def groups(out):
    return {ln["group"]: ln["items"] for ln in out["launches"] if ln["group"] >= 0}


def test_longest_items_first(batch):
    """A group's items are taken in order: a call whose long sectors come last must
    not end with their items."""
    out = batch("items", (4096, 0, 100, 2), (4096, 0, 3000, 3), (4096, 0, 900, 4),
                (16384, 1, 40, 3), (16384, 1, 500, 2))
    assert out["status"] == OK
    for items in groups(out).values():
        lengths = {}
        for scan, row, f0, f1, part, slots, flush in items:
            lengths.setdefault(scan, []).append(f1 - f0)
        longest = [max(v) for v in lengths.values()]  # in ticket order
        assert len(set(longest)) > 1 and longest == sorted(longest, reverse=True)


def test_many_short_sectors_run_whole(batch):
    """Where the sectors alone fill the GPU, a short one is one item with one partial
    slot; its f32 runs end at the same frames as its items do where it is split."""
    for fft, nf, few, many in ((1024, 400, 8, 2000), (4096, 150, 8, 1024), (8192, 75, 16, 512),
                               (16384, 40, 8, 256)):
        rows = 2 if fft == 16384 else 1
        split = batch("items", (fft, 0, nf, few))
        whole = batch("items", (fft, 0, nf, many))
        assert split["status"] == whole["status"] == OK
        (s_items,), (w_items,) = groups(split).values(), groups(whole).values()
        assert len(w_items) == many * rows and len(s_items) > 2 * few * rows
        assert all(f0 == 0 and f1 == nf and not slots for _, _, f0, f1, _, slots, _ in w_items)
        assert len({part for *_, part, _, _ in w_items}) == many  # rows share a slot
        fpc = {1024: 4}.get(fft, 1)
        lengths = {f1 - f0 for _, _, f0, f1, *_ in s_items if f1 < nf}
        assert lengths == {flush * fpc for *_, flush in w_items} and max(lengths) <= 32
        assert whole["in_use"] < 0.6 * many / few * split["in_use"]
    # sectors whose items have several runs stay split
    (items,) = groups(batch("items", (8192, 0, 2000, 512))).values()
    assert len(items) == 512 * 24


@pytest.mark.parametrize("sector,count,budget", [
    ((8192, 0, 100), 10, 1_600_000),     # a slot of 131 KB a sector and the tables
    ((8192, 0, 100), 40, 6_000_000),
    ((16384, 0, 100), 30, 10_000_000),
    ((1024, 0, 300), 500, 10_000_000),
    ((8192, 1, 64), 64, 2_500_000),
    ((4096, 0, 2000), 1, 1_500_000),     # one sector, items of several runs
    ((8192, 0, 100), 1, 200_000)])
def test_no_room_for_every_item(batch, sector, count, budget):
    """A call whose sectors' partials would fit unsplit is taken: fewer sectors at a
    time or, one alone, fewer items, its runs the same wherever an item has one."""
    out = batch("items", (*sector, count), budget=budget)
    assert out["status"] == OK and out["in_use"] <= budget
    fft, phased, nf = sector
    free = groups(batch("items", (*sector, 1)))
    fpc = {1024: 4}.get(fft, 1)
    one_run = max(f1 - f0 for items in free.values() for _, _, f0, f1, *_ in items) <= 32
    seen = 0
    for ln in out["launches"]:
        frames = {}
        for scan, row, f0, f1, part, slots, flush in ln["items"]:
            frames.setdefault((scan, row), []).append((f0, f1))
            if one_run:
                assert slots or f1 - f0 <= flush * fpc or (f0, f1) == (0, nf)
                assert flush == next(iter(free.values()))[0][-1]
        for (scan, row), f in frames.items():  # every frame once
            assert [a for a, _ in sorted(f)] == [0] + [b for _, b in sorted(f)][:-1]
            assert max(b for _, b in f) == nf
            seen += row == 0
    assert seen == count


def test_budget_too_small_stays_refused(batch):
    out = batch("items", (8192, 0, 100, 10), budget=100_000)
    assert out["status"] == EBUSY and not out["launches"]


@pytest.mark.parametrize("fail_at", range(5))
def test_launches_before_an_error_are_waited_for(batch, fail_at):
    """Records, three groups on streams of their own, reduction: when one of them fails,
    whatever was launched comes before the caller's next work on its stream and before
    the next call, on another stream."""
    out = batch("error", (1024, 0, 300, 3), (8192, 0, 100, 2), (8192, 1, 100, 1), fail_at=fail_at)
    assert out["status"] not in (OK, EBUSY) and out["again"] == OK
    launched = set(range(fail_at))
    assert out["stream"] == launched
    again = out["launches"][fail_at + 1:]
    assert again[0]["name"] == "records" and all(launched <= ln["before"] for ln in again)


def test_autotune_after_set_shape_splits_as_untouched(batch):
    """The tuner replaces a shape that the caller had pinned: short sectors are split by
    their own length again, as in a batch whose shape nobody has set."""
    pinned, free = (groups(batch(cmd, (8192, 0, 30, 1))) for cmd in ("pinned", "items"))
    assert len(free[3]) > 1 and [i[2:4] for i in pinned[3]] == [i[2:4] for i in free[3]]


@pytest.mark.parametrize("fft", [1024, 2048, 4096, 8192])
def test_runs_of_a_pinned_shape(batch, fft):
    """With one frame per iteration, whatever the scan's own kernel has, an f32 run is
    32 iterations."""
    (items,) = groups(batch("shape", (fft, 0, 300, 2))).values()
    assert {(f0 % 64, slots, flush) for _, _, f0, _, _, slots, flush in items} == {(0, 0, 32)}


def test_several_runs_an_item(batch):
    """Where the runs of FFT 1024..4096 are many, an item takes up to four in a row, each
    with the slot it has as an item of its own."""
    for fft, nf, many in ((1024, 300, 891), (2048, 130, 900), (4096, 150, 350)):
        (few,) = groups(batch("items", (fft, 0, nf, 1))).values()
        (items,) = groups(batch("items", (fft, 0, nf, many))).values()
        h = fft // 2 + 1
        run = few[0][3] - few[0][2]
        assert len(few) < len(items) < many * len(few)
        slots = {}
        for scan, row, f0, f1, part, own, flush in items:
            assert own and f0 % run == 0 and f1 - f0 <= 4 * run and flush == few[0][-1]
            for k in range(-(-(f1 - f0) // run)):
                slots.setdefault(scan, []).append((f0 + k * run, part + k * 4 * h))
        assert len(slots) == many
        for v in slots.values():  # the slots that single-run items have, in frame order
            base = min(p for _, p in v)
            assert sorted(v) == [(k * run, base + k * 4 * h) for k in range(len(few))]
