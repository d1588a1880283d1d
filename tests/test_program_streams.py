"""Launches of one program on several streams: they share its tables, staged copies, counters and workspace."""
import threading

import pytest
import torch

import universal_gemm_b200 as ug
from universal_gemm_b200.ops import fused, native

from helpers import make_inputs


class _Cuda:
    """The calls of torch.cuda that a program makes, written down."""

    def __init__(self):
        self.log, self.capturing, self.current = [], False, 0
        outer = self

        class Event:
            def record(self, stream):
                outer.log.append(("record", stream.raw))
                self.at = len(outer.log)

        class Stream:
            def __init__(self, raw, device=None):
                self.raw = self.cuda_stream = raw

            def wait_event(self, event):
                outer.log.append(("wait", self.raw, outer.log[event.at - 1][1]))

        self.Event, self.ExternalStream = Event, Stream
        self.default_stream = lambda device=None: Stream(0)
        self.current_stream = lambda device=None: Stream(self.current)
        self.is_current_stream_capturing = lambda: self.capturing


class _Memory:
    def __init__(self, log, name):
        self.log, self.name = log, name

    def record_stream(self, stream):
        self.log.append(("used", self.name, stream.raw))


@pytest.fixture
def cuda(monkeypatch):
    fake = _Cuda()
    monkeypatch.setattr(torch, "cuda", fake)
    return fake


def _program(cuda, built_on=0):
    cuda.current = built_on
    params = native.FusedParams()
    prog = fused.FusedProgram(device=torch.device("cuda", 0), tables=_Memory(cuda.log, "tables"), staging=None,
                              workspace=_Memory(cuda.log, "workspace"), params=params, grid=148, stats={})
    prog._entry = lambda ref, grid, stream: cuda.log.append(("launch", stream, params.checksum)) or 0

    def launch(stream, checksum=0):
        cuda.current = stream
        prog.launch(stream, checksum)
    return launch


def test_the_default_stream_alone_costs_no_event(cuda):
    launch = _program(cuda)
    launch(0), launch(0, 7), launch(0)
    assert cuda.log == [("launch", 0, 0), ("launch", 0, 7), ("launch", 0, 0)]


def test_a_launch_on_another_stream_waits_for_the_last_and_keeps_the_memory(cuda):
    launch = _program(cuda)
    launch(0), launch(5), launch(5), launch(9), launch(0)
    assert cuda.log == [("launch", 0, 0),
                        ("record", 0), ("wait", 5, 0), ("used", "tables", 5), ("used", "workspace", 5), ("launch", 5, 0), ("record", 5),
                        ("launch", 5, 0), ("record", 5),
                        ("wait", 9, 5), ("used", "tables", 9), ("used", "workspace", 9), ("launch", 9, 0), ("record", 9),
                        ("wait", 0, 9), ("used", "tables", 0), ("used", "workspace", 0), ("launch", 0, 0)]


def test_the_first_launch_waits_for_the_stream_that_built_the_tables(cuda):
    launch = _program(cuda, built_on=3)
    launch(0)
    assert cuda.log == [("record", 3), ("wait", 0, 3), ("used", "tables", 0), ("used", "workspace", 0), ("launch", 0, 0)]


def test_a_captured_launch_leaves_events_alone(cuda):
    """A captured stream must not wait for an event from outside, nor leave one behind."""
    launch = _program(cuda)
    cuda.capturing = True
    launch(5)
    cuda.capturing = False
    launch(0)
    assert cuda.log == [("launch", 5, 0), ("launch", 0, 0)]


def test_every_thread_s_launch_has_its_own_checksum(cuda):
    launch = _program(cuda)
    threads = [threading.Thread(target=lambda i=i: [launch(0, i) for _ in range(200)]) for i in range(1, 5)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert sorted(x[2] for x in cuda.log) == sorted([1, 2, 3, 4] * 200)


def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _zero_counters(prog):
    """Every word that a launch expects to be zero."""
    torch.cuda.synchronize()
    p, base = prog.params, prog._tables.data_ptr()
    words = [(p.flags, p.num_flags + 2 if p.num_pieces else 0), (p.part_flags, p.num_part_flags), (p.sched, 1 if p.sched else 0),
             (p.finished, 1 if p.finished else 0)]
    return all(int(prog._tables[at - base:at - base + 4 * n].view(torch.int32).abs().sum()) == 0 for at, n in words if n)


@pytest.mark.gpu
@pytest.mark.parametrize("tile_m", [128, 256, "pair"])
@pytest.mark.parametrize("staged", [False, True])
def test_launches_on_changing_streams(tile_m, staged):
    """Cut tiles and staged operands, launched in turn on three streams that nothing else orders: C += adds up."""
    from universal_gemm_b200.ops.device import DeviceState, torch_dtype_code
    from universal_gemm_b200.ops.gemm import _segments, _slice_of, run_program

    m, n, k = 300, 1030, 2304
    gen = torch.Generator(device=_dev()).manual_seed(3)
    a = torch.randn(m, k, device=_dev(), generator=gen).bfloat16()
    b = torch.zeros(k, 1088, device=_dev(), dtype=torch.bfloat16)[:, :n]
    b.copy_(torch.randn(k, n, device=_dev(), generator=gen) / k ** 0.5)
    c = torch.zeros(m, n, device=_dev())
    st = DeviceState.get(_dev())
    builder = fused.FusedProgramBuilder(_dev(), num_sms=st.num_sms, tile_m=tile_m, parts=3)
    builder.add_task(fused.TaskSpec(c_ptr=c.data_ptr(), ldc=n, m=m, n=n, c_mode=native.C_ADD, c_dtype=torch_dtype_code(c.dtype),
                                    segments=_segments(_slice_of(a, remote=staged), _slice_of(b, remote=staged))))
    prog = builder.build(st.status_ptr)
    streams = [torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.current_stream()]
    torch.cuda.synchronize()
    for i in range(30):
        with torch.cuda.stream(streams[i % 3]):
            run_program(prog, _dev())
    assert _zero_counters(prog)
    ug.check_status(_dev())
    want = 30 * (a.double() @ b.double())
    assert (c.double() - want).norm() <= 1e-5 * want.norm()


@pytest.mark.gpu
def test_a_program_dropped_while_another_stream_runs_it():
    """Its tables and staging area go back to the allocator only when that stream is done with them."""
    from universal_gemm_b200.parallel import exec as X

    m, n, k = 515, 700, 4100
    full_a, full_b, _ = make_inputs(m, n, k, seed=44, device=_dev())
    world = ug.EmulatedCluster(2, _dev()).worlds()
    mats = [(ug.distribute_tensor(full_a, w, "block", dtype=torch.bfloat16), ug.distribute_tensor(full_b, w, "row", dtype=torch.bfloat16),
             ug.zeros(w, (m, n), "column", torch.float32)) for w in world]
    side = torch.cuda.Stream()
    X.clear_program_cache()
    for a, b, c in mats:
        ug.matmul(a, b, c, method="stationary_c", beta=0)
    torch.cuda.synchronize()
    sizes = [(p._tables.numel(), p._staging.numel()) for _, p in X.cached_programs()]
    for _ in range(20):
        for a, b, c in mats:
            c.local_padded.zero_()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(4):
                for a, b, c in mats:
                    ug.matmul(a, b, c, method="stationary_c", beta=0)
        X.clear_program_cache()
        for pair in sizes:                       # would get the memory of a program that still runs
            for size in pair:
                torch.full((size,), 0xFF, dtype=torch.uint8, device=_dev())
        torch.cuda.current_stream().wait_stream(side)
        for a, b, c in mats:                     # lowered again, on the default stream
            ug.matmul(a, b, c, method="stationary_c", beta=0)
    torch.cuda.synchronize()
    ug.check_status(_dev())
    want = full_a.bfloat16().double() @ full_b.bfloat16().double()
    torch.testing.assert_close(mats[0][2].full_tensor().double(), want, rtol=2e-3, atol=2e-3)
    X.clear_program_cache()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tile_m", [(torch.bfloat16, "pair"), (torch.bfloat16, "128"), (torch.float32, "pair"), (torch.float32, "128")])
def test_counters_are_back_at_zero_after_replays(dtype, tile_m, monkeypatch):
    """Chunk counters, piece cursor, tile claim and finished workers of claimed (pair) and staged (fp32) programs, replayed
    from a graph on two streams that only the program orders, with an eager call between."""
    from universal_gemm_b200.parallel import exec as X

    monkeypatch.setenv("UGEMM_TILE_M", tile_m)
    m, n, k = 515, 2100, 2100
    full_a, full_b, _ = make_inputs(m, n, k, seed=43, device=_dev())
    world = ug.SingleWorld(_dev())
    a, b = ug.distribute_tensor(full_a, world, "row", dtype=dtype), ug.distribute_tensor(full_b, world, "column", dtype=dtype)
    c = ug.zeros(world, (m, n), "row", torch.float32)
    plan = ug.prepare_matmul(a, b, c, beta=0).capture()
    assert plan.program.params.finished != 0 or plan.program.params.sched == 0
    side = torch.cuda.Stream()
    for i in range(6):
        c.local_padded.fill_(9.0)
        torch.cuda.synchronize()
        plan()
        with torch.cuda.stream(side):
            plan()
        ug.matmul(a, b, c, beta=0)
        assert _zero_counters(plan.program)
    ug.check_status(_dev())
    want = full_a.to(dtype).double() @ full_b.to(dtype).double()
    assert (c.local.double() - want).norm() <= 3e-5 * want.norm()
    X.clear_program_cache()


@pytest.mark.gpu
def test_a_program_s_workspace_is_accounted_for_while_it_lives():
    from universal_gemm_b200.ops.device import DeviceState
    from universal_gemm_b200.ops.gemm import _segments, _slice_of

    st = DeviceState.get(_dev())
    a, b, c = (torch.zeros(256, 256, device=_dev(), dtype=d) for d in (torch.bfloat16, torch.bfloat16, torch.float32))
    before = fused._workspace_bytes.get(st.device.index, 0)
    builder = fused.FusedProgramBuilder(st.device, num_sms=st.num_sms, tile_m=128, parts=3)
    builder.add_task(fused.TaskSpec(c_ptr=c.data_ptr(), ldc=256, m=256, n=256, c_mode=native.C_STORE, c_dtype=native.DT_F32,
                                    segments=_segments(_slice_of(a), _slice_of(b))))
    prog = builder.build(st.status_ptr)
    assert fused._workspace_bytes[st.device.index] - before == prog._workspace.numel() * 4 >= 2 * 2 * 128 * 256 * 4
    del prog
    assert fused._workspace_bytes[st.device.index] == before


@pytest.mark.gpu
@pytest.mark.parametrize("tile_m", [128, 256, "pair"])
def test_counters_are_back_at_zero_after_a_launch_that_gave_up(tile_m):
    """A chunk counter that never gets there (one piece more than there are) runs into the launch's limit and reports a
    status; the launch after it starts from zero and is correct."""
    from universal_gemm_b200.ops.device import DeviceState, KernelStatusError
    from universal_gemm_b200.ops.gemm import build_gemm_program, run_program

    st = DeviceState.get(_dev())
    m, n, k = 300, 520, 700
    gen = torch.Generator(device=_dev()).manual_seed(12)
    a = torch.randn(m, k, device=_dev(), generator=gen).bfloat16()
    b = (torch.randn(k, n, device=_dev(), generator=gen) / k ** 0.5).bfloat16()
    c = torch.zeros(m, n, device=_dev())
    prog = build_gemm_program([a], [b], c, mode=native.C_STORE, tile_m=tile_m, stage_a=True, stage_b=True, timeout_ns=200_000_000)
    at = prog.params.flag_need - prog._tables.data_ptr()
    need = prog._tables[at:at + 4 * prog.params.num_flags].view(torch.int32)
    need += 1
    run_program(prog, _dev())
    torch.cuda.synchronize()
    with pytest.raises(KernelStatusError) as err:
        st.check()
    assert err.value.code in (native.ERR_TIMEOUT_FLAG, native.ERR_TIMEOUT_MBAR)
    assert _zero_counters(prog)
    need -= 1
    run_program(prog, _dev())
    ug.check_status(_dev())
    assert _zero_counters(prog)
    want = a.double() @ b.double()
    assert (c.double() - want).norm() <= 1e-5 * want.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["stationary_b", "stationary_c"])
@pytest.mark.parametrize("triple", [("row", "column", "row"), ("block", "row", "column"), ("column", "block", "block")])
@pytest.mark.parametrize("tile_m", ["128", "256", "pair"])
@pytest.mark.parametrize("c_dtype", [torch.float32, torch.bfloat16])
def test_cut_tiles_on_several_ranks_stay_inside_their_allocations(method, triple, tile_m, c_dtype, monkeypatch):
    """Every tile of every rank in three K parts, through ug.matmul: operands staged from peers in several K ranges, results
    pushed into peers; guard regions around every tile."""
    from helpers import build_cluster_matrices
    from universal_gemm_b200.parallel import exec as X

    init = fused.FusedProgramBuilder.__init__
    monkeypatch.setattr(fused.FusedProgramBuilder, "__init__",
                        lambda self, *args, **kw: init(self, *args, **dict(kw, split_k=False, parts=3)))
    monkeypatch.setenv("UGEMM_TILE_M", tile_m)
    m, n, k = 301, 403, 1900
    full_a, full_b, full_c = make_inputs(m, n, k, seed=21, device=_dev())
    cluster = ug.EmulatedCluster(4, _dev(), guard_bytes=4096)
    mats = build_cluster_matrices(cluster, full_a, full_b, full_c, triple, 1, torch.bfloat16, c_dtype)
    X.clear_program_cache()
    for a, b, c in mats:
        ug.matmul(a, b, c, method=method)
    ug.check_status(_dev())
    assert cluster.check_guards() == 12
    progs = [p for _, p in X.cached_programs()]
    assert progs and all(p.stats["parts"] == 3 and p.stats["cut_tiles"] > 0 for p in progs)
    want = full_c.to(c_dtype).double() + full_a.bfloat16().double() @ full_b.bfloat16().double()
    # bf16: as many roundings of a sum of two as ranks add into an element (four), 2^-8 each for the share and the result
    tol = 1e-4 if c_dtype == torch.float32 else 4 * 2.0 ** -8
    assert ((mats[0][2].full_tensor().double() - want).abs() <= tol * (1.0 + want.abs())).all()
    X.clear_program_cache()


@pytest.mark.gpu
def test_matrices_made_again_at_old_addresses():
    """Clusters made and dropped in turn, of both result types and with one matrix kept over: every call runs a program of
    its own matrices, and the dropped ones' programs are gone."""
    import gc

    from helpers import build_cluster_matrices
    from universal_gemm_b200.parallel import exec as X

    m, n, k = 301, 403, 700
    full_a, full_b, full_c = make_inputs(m, n, k, seed=22, device=_dev())
    prod = full_a.bfloat16().double() @ full_b.bfloat16().double()
    X.clear_program_cache()
    kept = []
    for i in range(12):
        cluster = ug.EmulatedCluster(2 + 2 * (i % 2), _dev())
        dtype = (torch.float32, torch.bfloat16)[i // 2 % 2]
        mats = build_cluster_matrices(cluster, full_a, full_b, full_c, ("block", "row", "column"), 1, torch.bfloat16, dtype)
        if i % 3 == 1:                                       # peers' tiles move, this rank's may not
            kept = [torch.empty(mats[0][0].nbytes, dtype=torch.uint8, device=_dev()) for _ in range(i)]
        for a, b, c in mats:
            ug.matmul(a, b, c, method="stationary_c")
        ug.check_status(_dev())
        want = full_c.to(dtype).double() + prod
        tol = 1e-4 if dtype == torch.float32 else 2 * 2.0 ** -8
        assert ((mats[0][2].full_tensor().double() - want).abs() <= tol * (1.0 + want.abs())).all()
        assert len(X.cached_programs()) == len(mats)
        del cluster, mats, a, b, c
        gc.collect()
        assert not X.cached_programs()
