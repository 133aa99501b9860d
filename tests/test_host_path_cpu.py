"""What the library asks of the CUDA runtime, on a runtime made for the purpose
(tests/cpp/fake_cudart.cpp): no GPU, no kernel runs."""
import os
import subprocess

import pytest

from conftest import ROOT, pkg

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    lib = pkg("_lib").LIB_PATH
    if not os.path.exists(lib):
        pkg("build").build()
    out = str(tmp_path_factory.mktemp("fake") / "fake_cudart")
    libdir = os.path.dirname(lib)
    subprocess.run(["g++", "-std=c++17", "-O1", "-rdynamic", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(CUDA, "include"),
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), "-L", libdir,
                    "-lmdgemm", "-Wl,-rpath," + libdir, "-Wl,--allow-shlib-undefined", "-o", out],
                   check=True, capture_output=True)

    def run(*words, **env):
        r = subprocess.run([out] + [str(w) for w in words], capture_output=True, text=True,
                           timeout=120, env={**os.environ, **env})
        assert r.returncode == 0, r.stderr[-2000:]
        return [line.split() for line in r.stdout.splitlines()]

    return run


def _statuses(lines):
    return [int(line[2]) for line in lines if line[0] == "status"]


def test_a_kernels_shared_memory_limit_is_the_same_at_every_call(fake):
    """The limit belongs to the kernel and all host threads share it: one that
    set its own call's size would have the launches of others refused."""
    words = []
    for p in (2, 4, 8, 16):
        for shape in ((64, 64, 64), (256, 100, 90), (1024, 1024, 512), (600, 700, 1024),
                      (3000, 64, 100), (900, 900, 20000)):
            words += ["gemm", 2, p, *shape]
        words += ["batch", p, 64, 96, 65, "batched", 0, p, 10, 20, 30, "gemm", 3, p, 50, 60, 70,
                  "gemm", 0, p, 50, 60, 70]
    words += ["digits", 119, 112, "gemm", 2, 16, 64, 64, 64, "gemm", 2, 16, 1024, 1024, 1024]
    words += ["gemm", 2, 16, 1024, 1024, 20000]
    # 48 rows of 1 KiB in the sums kernel: the default limit without static memory
    words += ["digits", 48, 48, "gemm", 2, 4, 1024, 1024, 1024]
    lines = fake(*words)
    assert set(_statuses(lines)) == {0}
    limits, launches = {}, {}
    for line in lines:
        if line[0] == "limit":
            limits.setdefault(line[1], set()).add(int(line[2]))
        elif line[0] == "launch":
            launches[line[1]] = max(launches.get(line[1], 0), int(line[2]))
            assert int(line[2]) <= 47 * 1024 or previous[:2] == ["limit", line[1]]
        previous = line
    assert len(limits) >= 8 and len(launches) >= 20
    assert {k: v for k, v in limits.items() if len(v) > 1} == {}
    for kernel, smem in launches.items():
        assert smem <= max(limits.get(kernel, {47 * 1024})), kernel
    assert max(max(v) for v in limits.values()) <= 227 * 1024


@pytest.mark.parametrize("p,m,n,k,operands", [
    (4, 1024, 1024, 1024, 3 << 25),      # one workspace, 1.1 GiB with the sum planes
    (2, 2048, 256, 300, 0),              # row panels: nothing to fall back to
])
def test_host_entry_after_an_allocation_that_failed(fake, p, m, n, k, operands):
    """A workspace with sum planes that the device has no room for: the call
    runs over digit pairs, and the failed allocation's error is not taken for
    that of a launch.  Without room for those either, the call says so and the
    next one that fits succeeds."""
    least = pkg("_lib").lib().mdg_gemm_least_workspace_size(2, p, m, n, k, None)
    if operands:
        lines = fake("capacity", operands + least, "host", p, m, n, k)
        assert ["oom"] in [line[:1] for line in lines] and _statuses(lines) == [0]
    lines = fake("capacity", 24 << 20, "host", p, m, n, k, "host", 2, 32, 32, 32, "plan", p, m, n, k,
                 "gemm", 2, 2, 32, 32, 32)
    assert _statuses(lines) == [9, 0, 9, 0]  # 9: allocation failed


def test_host_entry_gives_back_memory_that_it_does_not_use(fake):
    """Two column strips.  Room for one strip's sum planes but not for two:
    both strips run over digit pairs, in the room the first one had.  And a
    call that finds the device filled by an earlier call's workspaces."""
    p, m, n, k = 2, 2048, 4096, 1024
    operands = 8 * p * (m * k + k * n + m * n)
    sums = [int(line[1]) for line in fake("host", p, m, n, k) if line[0] == "malloc"][3:]
    pairs = pkg("_lib").lib().mdg_gemm_least_workspace_size(2, p, 1024, 2048, k, None)
    assert len(sums) == 2 and sums[0] + pairs > sums[0] + (16 << 20) > 2 * pairs
    room = operands + sums[0] + (16 << 20)
    lines = fake("capacity", room, "host", p, m, n, k)
    assert _statuses(lines) == [0]
    assert [int(line[1]) for line in lines if line[0] == "malloc"][-2:] == [pairs, pairs]
    lines = fake("host", p, m, n, k, "capacity", room + (1 << 20), "host", p, m, n + 8, k)
    assert _statuses(lines) == [0, 0]


def _schedules(lines):
    return [tuple(int(v) for v in line[3:]) for line in lines if line[0] == "status"
            and line[1] in ("plan", "tune")]


@pytest.mark.parametrize("p,m,n,k,wide_m,wide_n", [
    (2, 16001, 96, 3001, 16001, 256),   # two diagonals an accumulator
    (8, 100, 20000, 100, 256, 20000),
    (4, 100, 100, 500, 256, 256),       # tiles of 128 columns
])
def test_tuning_can_keep_the_automatic_tiles(fake, tmp_path, p, m, n, k, wide_m, wide_n):
    """The runtime times tiles that only the automatic engine has as the fastest:
    a tuned plan keeps them, later plans of the shape too, and records of the
    padded sizes (older files, wider problems) do not apply to it."""
    import json
    own, wide = (p, m, n, k), (p, wide_m, wide_n, k)
    out = tmp_path / "tune.json"
    lines = fake("tune", *own, "plan", *own, "plan", *wide, "save", out)
    assert _schedules(lines) == [(0, 0, 0, 0)] * 3
    key = list(json.loads(out.read_text())["fake|1"])
    assert len(key) == 1
    old = tmp_path / "old.json"
    padded = " ".join(key[0].split()[:7])
    assert padded != key[0]
    old.write_text(json.dumps({"fake|1": {padded: {"engine": 1, "parts": 2, "raster": 0,
                                                   "pace": 0, "ms": 1.0}}}))
    assert _schedules(fake("load", old, "plan", *own, "plan", *wide)) == [(0,) * 4, (1, 2, 0, 0)]


def test_tuning_of_ordinary_shapes_picks_an_engine(fake):
    lines = fake("tune", 4, 1024, 768, 512, "plan", 4, 1000, 700, 500)
    assert _schedules(lines) == [(2, 0, 0, 0)] * 2


@pytest.mark.parametrize("shape", [(4, 1024, 1024, 1024), (2, 16001, 96, 3001)])
def test_pacing_window_of_the_environment(fake, shape):
    """MDG_TC_PACE sets the window on the launches whose units would otherwise be
    dealt by cost, as mdg_options.pace does; 0 and no value leave them dealt."""
    def schedules(**env):
        lines = [line[3:] for line in fake("gemm", 2, *shape, **env)
                 if line[0] == "launch" and line[1].startswith("diag_gemm")]
        return [dict(word.split("=") for word in line) for line in lines]

    for env in ({}, {"MDG_TC_PACE": "0"}):
        for s in schedules(**env):
            assert (s["pace"], s["dealt"]) == ("0", "1"), env
    for s in schedules(MDG_TC_PACE="96"):
        assert (s["pace"], s["dealt"]) == ("96", "0")


@pytest.mark.parametrize("m,n,columns", [(512, 512, 2), (256, 512, 2), (255, 512, 1),
                                         (512, 513, 1), (700, 900, 2)])
def test_renormalisation_takes_two_columns_a_thread(fake, m, n, columns):
    """From 2^17 entries on, where rows of the chunk planes are aligned for it."""
    for p in (2, 4, 8):
        names = [line[1] for line in fake("renorm", p, m, n, 500) if line[0] == "launch"]
        assert names == [f"renorm_kernelILi{columns}EEE"]


@pytest.mark.parametrize("m,n,k", [(256, 256, 256), (500, 500, 70)])
def test_host_time_of_a_dealt_call(fake, m, n, k):
    """The host deals the units of a hexa-double problem of few tiles in a walk
    over its runs (a few times the cost of one that is not dealt), not in a walk
    a part (eight and more times)."""
    import time

    def seconds(calls, *shape):
        best = 1e9
        for _ in range(5):
            t = time.perf_counter()
            fake(*(["gemm", 2, 16, *shape] * calls))
            best = min(best, time.perf_counter() - t)
        return best

    plain, dealt = (seconds(1501, *s) - seconds(1, *s) for s in ((64, 64, 64), (m, n, k)))
    assert dealt < 4.5 * plain, (dealt, plain)


def test_the_smaller_workspace_is_asked_for_when_memory_is_short(monkeypatch):
    """api.gemm's workspace: what the call can do without is worked out only after
    an allocation failed."""
    import torch
    api = pkg("api")
    ws, got = api._workspace(4096, lambda: pytest.fail("memory was there"), "cpu")
    assert (ws.numel(), got) == (4096, 4096)
    empty = torch.empty

    def short(n, **kw):
        if n > 3000:
            raise torch.OutOfMemoryError("short")
        return empty(n, **kw)

    monkeypatch.setattr(api.torch, "empty", short)
    ws, got = api._workspace(4096, lambda: 1096, "cpu")
    assert (ws.numel(), got) == (3000, 3000)
    with pytest.raises(torch.OutOfMemoryError):
        api._workspace(4096, lambda: 0, "cpu")


@pytest.mark.parametrize("p,m,n,k", [(2, 40, 40, 40), (8, 500, 300, 200), (16, 2000, 1500, 100)])
def test_a_captured_batch_finds_its_units_after_the_split_mode_changed(fake, p, m, n, k):
    """A graph captured with heavy tiles split, replayed after mdg_batch_set_split(0):
    the launch it holds takes each of the new table's units (tiles) once."""
    lines = fake("batch", p, m, n, k)
    assert _statuses(lines) == [0]
    units = [int(u) for line in lines if line[0] == "replay" for u in line[1:]]
    assert sorted(units) == list(range(-(-m // 128) * -(-n // 256)))


def test_a_callers_workspace_without_room_for_sum_planes_is_used():
    """One made for the digit pairs, as mdg_gemm takes it; a smaller one is not."""
    import torch
    api = pkg("api")
    for size, used in ((8000, 4096), (4096, 4096), (3500, 3500), (3000, 3000)):
        given = torch.empty(size, dtype=torch.uint8)
        ws, got = api._workspace(4096, lambda: 1096, "cpu", given)
        assert ws is given and got == used
    given = torch.empty(2999, dtype=torch.uint8)
    ws, got = api._workspace(4096, lambda: 1096, "cpu", given)
    assert ws is not given and ws.numel() == got == 4096


@pytest.mark.gpu
def test_gemm_in_a_callers_workspace_for_digit_pairs():
    import torch
    api, L = pkg("api"), pkg("_lib").lib()
    p, n = 4, 1024
    A, B = api.generate("uniform", p, n, n, 1), api.generate("uniform", p, n, n, 2)
    ref = api.gemm(A, B)
    ws = torch.empty(L.mdg_gemm_least_workspace_size(2, p, n, n, n, None), dtype=torch.uint8,
                     device="cuda")
    out = torch.empty_like(ref)
    free = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    api.gemm(A, B, out=out, workspace=ws)
    assert torch.cuda.max_memory_allocated() == free and torch.equal(out, ref)
    ex = api.gemm_ex(A, B.transpose(0, 1).contiguous(), trans_b=True, C=out, workspace=ws)
    assert torch.equal(ex, ref)
