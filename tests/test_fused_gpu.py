"""GPU tests: the fused tcgen05 kernel and the tile kernels against fp32 PyTorch references,
and the fused executors on an emulated multi-rank cluster that lives on one GPU (ranks run
one after the other; remote tiles are other buffers of the same GPU, so every fetch / push
path of the kernel is exercised without a second device)."""
import pytest
import torch

import universal_gemm_b200 as ug

from helpers import ALL_TRIPLES, build_cluster_matrices, make_inputs, oracle, run_cluster

pytestmark = pytest.mark.gpu


def _dev():
    return torch.device("cuda", 0)


def _status_ok():
    from universal_gemm_b200.ops.device import DeviceState

    torch.cuda.synchronize()
    DeviceState.get(_dev()).check()


def _native_loaded():
    from universal_gemm_b200.ops import build

    with open("/proc/self/maps") as f:
        return str(build.library_path()) in f.read()


def test_native_library_is_loaded():
    from universal_gemm_b200.ops import native

    assert native.lib().ug_version() >= 1
    assert _native_loaded()


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (512, 1024, 512), (300, 520, 200), (375, 1000, 376),
                                   (64, 4099, 1024), (2048, 4096, 1024), (1, 8, 8)])
@pytest.mark.parametrize("mode", ["store", "add", "atomic"])
@pytest.mark.parametrize("tile_m", [128, 256, "pair", "pair512"])
def test_gemm_kernel_fp32_out(m, n, k, mode, tile_m):
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import gemm

    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device=_dev()).bfloat16()
    b = (torch.randn(k, n, device=_dev()) / k ** 0.5).bfloat16()
    c0 = torch.randn(m, n, device=_dev())
    c = c0.clone()
    gemm(a, b, c, mode={"store": native.C_STORE, "add": native.C_ADD, "atomic": native.C_ATOMIC}[mode], tile_m=tile_m)
    _status_ok()
    ref = a.float() @ b.float() + (0 if mode == "store" else c0)
    torch.testing.assert_close(c, ref, rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("mode", ["store", "add", "atomic"])
def test_gemm_kernel_bf16_out(mode):
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import gemm

    torch.manual_seed(5)
    m, n, k = 384, 777, 320
    a = torch.randn(m, k, device=_dev()).bfloat16()
    b = (torch.randn(k, n, device=_dev()) / k ** 0.5).bfloat16()
    c0 = torch.randn(m, n, device=_dev()).bfloat16()
    c = c0.clone()
    gemm(a, b, c, mode={"store": native.C_STORE, "add": native.C_ADD, "atomic": native.C_ATOMIC}[mode])
    _status_ok()
    ref = a.float() @ b.float() + (0 if mode == "store" else c0.float())
    torch.testing.assert_close(c.float(), ref, rtol=2e-2, atol=3e-2)


@pytest.mark.parametrize("stage_a,stage_b", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("tile_m", [128, 256, "pair", "pair512"])
def test_gemm_kernel_segments_and_staging(stage_a, stage_b, tile_m):
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import build_gemm_program, run_program

    torch.manual_seed(9)
    m, n, k = 640, 1290, 1500
    a = torch.randn(m, k, device=_dev()).bfloat16()
    b = (torch.randn(k, n, device=_dev()) / k ** 0.5).bfloat16()
    c = torch.zeros(m, n, device=_dev())
    cuts = [0, 500, 1001, 1500]          # 1001 is not a multiple of 8: that segment is staged and re-aligned
    prog = build_gemm_program([a[:, cuts[i]:cuts[i + 1]] for i in range(3)], [b[cuts[i]:cuts[i + 1]] for i in range(3)],
                              c, mode=native.C_STORE, stage_a=stage_a, stage_b=stage_b, tile_m=tile_m)
    assert prog.num_pieces > 0
    for _ in range(2):                   # second launch checks that the counters are reset
        run_program(prog, _dev())
    _status_ok()
    torch.testing.assert_close(c, a.float() @ b.float(), rtol=2e-3, atol=2e-3)


def test_tile_kernels():
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.device import DeviceState

    st = DeviceState.get(_dev())
    torch.manual_seed(0)
    for dtype, code in ((torch.float32, native.DT_F32), (torch.bfloat16, native.DT_BF16)):
        es = torch.empty(0, dtype=dtype).element_size()
        for rows, cols, off in ((64, 128, 0), (37, 53, 0), (37, 53, 3), (1, 8, 0)):
            src = torch.randn(rows + 2, cols + 16, device=_dev()).to(dtype)
            dst = torch.zeros(rows + 2, cols + 24, device=_dev(), dtype=dtype)
            sv, dv = src[1:1 + rows, off:off + cols], dst[1:1 + rows, 8:8 + cols]
            st.pull_2d(dv.data_ptr(), dst.stride(0) * es, sv.data_ptr(), src.stride(0) * es, rows, cols * es, es)
            torch.cuda.synchronize()
            outside = dst.clone()
            outside[1:1 + rows, 8:8 + cols] = 0
            assert torch.equal(dv, sv) and outside.abs().max().item() == 0
            before = dv.clone()
            st.accumulate_2d(dv.data_ptr(), dst.stride(0), sv.data_ptr(), src.stride(0), rows, cols, code)
            torch.cuda.synchronize()
            torch.testing.assert_close(dv.float(), before.float() * 2, rtol=1e-2, atol=1e-2)
            st.zero_2d(dv.data_ptr(), dst.stride(0) * es, rows, cols * es)
            torch.cuda.synchronize()
            assert dst.abs().sum() == 0
    f = torch.randn(33, 47, device=_dev())
    h = torch.zeros(33, 64, device=_dev(), dtype=torch.bfloat16)
    st.convert_2d(h.data_ptr(), 64, native.DT_BF16, f.data_ptr(), 47, native.DT_F32, 33, 47)
    torch.cuda.synchronize()
    assert torch.equal(h[:, :47], f.bfloat16())
    f2 = torch.randn(40, 96, device=_dev())                       # aligned: the 16-byte vector kernels
    h2 = torch.zeros(40, 128, device=_dev(), dtype=torch.bfloat16)
    st.convert_2d(h2.data_ptr(), 128, native.DT_BF16, f2.data_ptr(), 96, native.DT_F32, 40, 96)
    back = torch.zeros(40, 96, device=_dev())
    st.convert_2d(back.data_ptr(), 96, native.DT_F32, h2.data_ptr(), 128, native.DT_BF16, 40, 96)
    torch.cuda.synchronize()
    assert torch.equal(h2[:, :96], f2.bfloat16()) and torch.equal(back, f2.bfloat16().float()) and h2[:, 96:].abs().sum() == 0


@pytest.mark.parametrize("world,rep", [(1, 1), (2, 1), (4, 2), (8, 1), (8, 2), (8, 4)])
@pytest.mark.parametrize("method", ["stationary_c", "stationary_b"])
def test_fused_all_triples_emulated(world, rep, method):
    m, n, k = 301, 203, 157
    full_a, full_b, full_c = make_inputs(m, n, k, seed=world + rep, device=_dev())
    triples = ALL_TRIPLES if world == 8 and rep == 1 else ALL_TRIPLES[::3]
    for triple in triples:
        cluster = ug.EmulatedCluster(world, _dev())
        mats = build_cluster_matrices(cluster, full_a, full_b, full_c, triple, rep, torch.bfloat16, torch.float32)
        run_cluster(cluster, mats, method, executor="fused")
        _status_ok()
        got = mats[0][2].full_tensor(replica=0)
        torch.testing.assert_close(got.double(), oracle(full_a, full_b, full_c, torch.bfloat16), rtol=2e-3, atol=2e-3,
                                   msg=lambda s: f"{method} {triple} world={world} rep={rep}: {s}")


@pytest.mark.parametrize("triple", [("row", "row", "row"), ("row", "column", "row"), ("column", "row", "row"),
                                    ("block", "block", "block")])
@pytest.mark.parametrize("method", ["stationary_c", "stationary_b", "auto"])
def test_fused_medium_shapes_emulated(triple, method):
    m, n, k = 1024, 1536, 2048
    full_a, full_b, full_c = make_inputs(m, n, k, seed=11, device=_dev())
    for rep, out_dtype in ((1, torch.float32), (2, torch.float32), (1, torch.bfloat16)):
        cluster = ug.EmulatedCluster(8, _dev())
        mats = build_cluster_matrices(cluster, full_a, full_b, full_c, triple, rep, torch.bfloat16, out_dtype)
        for _ in range(2):
            run_cluster(cluster, mats, method, executor="fused")
        _status_ok()
        got = mats[0][2].full_tensor(replica=0).double()
        want = full_c.to(out_dtype).double() + 2 * (full_a.bfloat16().double() @ full_b.bfloat16().double())
        tol = 3e-3 if out_dtype == torch.float32 else 6e-2
        torch.testing.assert_close(got, want, rtol=tol, atol=tol,
                                   msg=lambda s: f"{method} {triple} rep={rep} {out_dtype}: {s}")


def test_unfused_replica_reduce_and_tilewise_on_gpu():
    m, n, k = 256, 320, 512
    full_a, full_b, full_c = make_inputs(m, n, k, seed=2, device=_dev())
    for executor in ("fused", "tilewise"):
        cluster = ug.EmulatedCluster(4, _dev())
        mats = build_cluster_matrices(cluster, full_a, full_b, full_c, ("row", "row", "row"), 2, torch.bfloat16,
                                      torch.float32)
        run_cluster(cluster, mats, "stationary_c", executor=executor, fuse_replica_reduce=False)
        _status_ok()
        torch.testing.assert_close(mats[0][2].full_tensor().double(), oracle(full_a, full_b, full_c, torch.bfloat16),
                                   rtol=3e-3, atol=3e-3)


def test_tile_api_on_gpu():
    cluster = ug.EmulatedCluster(4, _dev())
    full = torch.randn(64, 48, device=_dev())
    mats = [ug.distribute_tensor(full, w, "row") for w in cluster.worlds()]
    dm = mats[1]
    ug.init_scratch(4 * 16 * 64, torch.float32, world=dm.world)
    t = ug.get_tile(dm, (3, 0))
    fut = ug.get_tile_async(dm, (0, 0), region=ug.Slice2D(ug.Slice1D(3, 9), ug.Slice1D(5, 40)))
    part = fut.get()
    torch.cuda.synchronize()
    assert torch.equal(t, full[48:64]) and torch.equal(part, full[3:9, 5:40])
    ug.release_tile(t)
    ug.accumulate_tile(dm, (2, 0), torch.ones(16, 48, device=_dev())).wait()
    torch.testing.assert_close(mats[2].local, full[32:48] + 1)
    ug.free_get_tile_scratch()


def test_bounded_wait_reports_timeout_instead_of_hanging():
    """A cross-rank barrier whose peer never signals runs out after its limit and reports a
    status code; the context stays usable."""
    import ctypes

    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.device import DeviceState, KernelStatusError

    st = DeviceState.get(_dev())
    slots = torch.zeros(2, 8, dtype=torch.int32, device=_dev())      # "rank 1" never adds to our slot
    table = torch.tensor([slots[0].data_ptr(), slots[1].data_ptr()], dtype=torch.int64, device=_dev())
    rounds = torch.zeros(1, dtype=torch.int32, device=_dev())
    native.check(native.lib().ug_signal_barrier(table.data_ptr(), 2, 0, rounds.data_ptr(), st.status_ptr, 50_000_000,
                                                ctypes.c_void_p(st.stream())), "ug_signal_barrier")
    torch.cuda.synchronize()
    with pytest.raises(KernelStatusError) as err:
        st.check()
    assert err.value.code == native.ERR_TIMEOUT_PEER
    assert slots[1, 0].item() == 1 and rounds.item() == 1             # our own signal was delivered
    st.check()                                                        # status cleared, context alive
    assert torch.ones(4, device=_dev()).sum().item() == 4


@pytest.mark.parametrize("method,triple", [("stationary_c", ("row", "row", "row")), ("stationary_c", ("block", "column", "block")),
                                           ("stationary_b", ("row", "column", "row")), ("stationary_b", ("block", "column", "row"))])
def test_beta_zero_overwrites_without_zeroing(method, triple):
    """beta=0 on single-writer plans stores C = A @ B whatever C held before (no zeroing pass)."""
    m, n, k = 520, 390, 450
    full_a, full_b, full_c = make_inputs(m, n, k, seed=4, device=_dev())
    cluster = ug.EmulatedCluster(4, _dev())
    mats = build_cluster_matrices(cluster, full_a, full_b, full_c * 100, triple, 1, torch.bfloat16, torch.float32)
    for a, b, c in mats:
        ug.matmul(a, b, c, method=method, beta=0)
    _status_ok()
    want = full_a.bfloat16().double() @ full_b.bfloat16().double()
    torch.testing.assert_close(mats[0][2].full_tensor().double(), want, rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("tile_m,m,n", [("pair", 512, 10240 - 17), (256, 512, 19712 - 5), (128, 256, 19712),
                                        ("pair512", 512, 20480 - 17)])
def test_gemm_kernel_tail_wave_uses_narrow_tiles(tile_m, m, n):
    """Tile counts just above a multiple of the worker count: the trailing tile columns run as 128-wide tiles."""
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import build_gemm_program, run_program

    torch.manual_seed(n)
    k = 320
    a = torch.randn(m, k, device=_dev()).bfloat16()
    b = (torch.randn(k, n, device=_dev()) / k ** 0.5).bfloat16()
    c = torch.full((m, n), 3.0, device=_dev())
    prog = build_gemm_program([a], [b], c, mode=native.C_ADD, tile_m=tile_m)
    assert prog.stats["tasks"] == 2                      # the task was split into a wide and a narrow part
    run_program(prog, _dev())
    _status_ok()
    torch.testing.assert_close(c, a.float() @ b.float() + 3.0, rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("method", ["stationary_b", "stationary_c"])
def test_fused_tail_split_with_remote_tiles(method, monkeypatch):
    """Two emulated ranks with 80 tiles each on 74 CTA pairs: the last three tile columns run as narrow tiles,
    with the A slices staged from the 'peer' and (Stationary-B) the result stored into the peer's C."""
    from universal_gemm_b200.parallel import exec as X

    monkeypatch.setenv("UGEMM_TILE_M", "pair")
    m, n, k = 1024, 10240, 256
    full_a, full_b, full_c = make_inputs(m, n, k, seed=6, device=_dev())
    cluster = ug.EmulatedCluster(2, _dev())
    mats = build_cluster_matrices(cluster, full_a, full_b, full_c, ("row", "column", "row"), 1, torch.bfloat16,
                                  torch.float32)
    X.clear_program_cache()
    for a, b, c in mats:
        ug.matmul(a, b, c, method=method, beta=0)
    _status_ok()
    stats = [v[2][0].stats for v in X._program_cache.values()]
    assert all(s["tiles"] == 86 and s["tasks"] == 3 for s in stats), stats   # 74 wide + 12 narrow tiles
    want = full_a.bfloat16().double() @ full_b.bfloat16().double()
    torch.testing.assert_close(mats[0][2].full_tensor().double(), want, rtol=2e-3, atol=2e-3)
    X.clear_program_cache()


def test_redistribute_on_gpu():
    full = torch.randn(301, 203, device=_dev())
    cluster = ug.EmulatedCluster(4, _dev())
    srcs = [ug.distribute_tensor(full, w, "block") for w in cluster.worlds()]
    outs = [ug.redistribute(s, "column") for s in srcs]
    halves = [ug.redistribute(s, "row", dtype=torch.bfloat16) for s in srcs]
    torch.cuda.synchronize()
    assert torch.equal(outs[2].full_tensor(), full)
    assert torch.equal(halves[1].full_tensor().float(), full.bfloat16().float())


def test_prepared_matmul_and_cuda_graph():
    """A prepared plan gives the same result eagerly and when replayed from a CUDA graph."""
    m, n, k = 512, 768, 640
    full_a, full_b, full_c = make_inputs(m, n, k, seed=12, device=_dev())
    world = ug.SingleWorld(_dev())
    a = ug.distribute_tensor(full_a, world, "row", dtype=torch.bfloat16)
    b = ug.distribute_tensor(full_b, world, "column", dtype=torch.bfloat16)
    c = ug.distribute_tensor(full_c, world, "row", dtype=torch.float32)
    plan = ug.prepare_matmul(a, b, c, method="stationary_c", beta=1)
    plan.run()
    _status_ok()
    prod = full_a.bfloat16().double() @ full_b.bfloat16().double()
    torch.testing.assert_close(c.full_tensor().double(), full_c.double() + prod, rtol=2e-3, atol=2e-3)
    plan.capture(warmup=1)              # two more accumulations: warm-up + capture run nothing new... capture does not execute
    torch.cuda.synchronize()
    before = c.full_tensor().double()
    for _ in range(3):
        plan()
    _status_ok()
    torch.testing.assert_close(c.full_tensor().double(), before + 3 * prod, rtol=2e-3, atol=4e-3)


@pytest.mark.parametrize("tile_m", [128, 256, "pair", "pair512"])
def test_kernel_timeline_records_every_tile(tile_m):
    """With tracing on, every tile leaves a record whose stamps are ordered, the fetch warps account for every
    staged piece, and the result is unchanged."""
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import build_gemm_program, run_program
    from universal_gemm_b200.utils import trace as TR

    torch.manual_seed(21)
    m, n, k = 1024, 1536, 768
    a = torch.randn(m, k, device=_dev()).bfloat16()
    b = (torch.randn(k, n, device=_dev()) / k ** 0.5).bfloat16()
    c = torch.zeros(m, n, device=_dev())
    prog = build_gemm_program([a], [b], c, mode=native.C_STORE, stage_a=True, tile_m=tile_m)
    assert prog.read_trace() is None
    prog.enable_trace()
    run_program(prog, _dev())
    _status_ok()
    torch.testing.assert_close(c, a.float() @ b.float(), rtol=2e-3, atol=2e-3)
    arr = prog.read_trace()
    pair = str(tile_m).startswith("pair")
    slots = arr.shape[1] - 1
    tiles = arr[:, :slots]
    leaders = tiles[::2] if pair else tiles
    seen = sorted(int(t) - 1 for t in leaders[:, :, TR.TILE].ravel() if t > 0)
    assert seen == list(range(prog.stats["tiles"]))
    rec = leaders[leaders[:, :, TR.TILE] > 0]
    assert (rec[:, TR.PROD_BEGIN] <= rec[:, TR.PROD_END]).all()
    assert (rec[:, TR.MMA_BEGIN] <= rec[:, TR.MMA_ISSUED]).all() and (rec[:, TR.MMA_BEGIN] > 0).all()
    assert (rec[:, TR.MMA_BEGIN] <= rec[:, TR.EPI_BEGIN]).all() and (rec[:, TR.EPI_BEGIN] <= rec[:, TR.EPI_END]).all()
    summ = arr[:, slots]
    assert (summ[:, TR.S_START] > 0).all() and (summ[:, TR.S_END] >= summ[:, TR.S_START]).all()
    assert int(summ[:, TR.S_PIECES].sum()) == prog.num_pieces
    s = TR.summarize(arr, pair=pair)
    assert s["recorded_tiles"] == prog.stats["tiles"] and s["pieces_copied"] == prog.num_pieces
    assert 0 < s["main_us_mean"] < s["kernel_us"] < 1e5
    assert 0.1 < s["sm_clock_ghz"] < 3.0               # SM cycles per globaltimer nanosecond
    assert TR.to_chrome_trace(arr)
    prog.disable_trace()
    run_program(prog, _dev())
    _status_ok()


@pytest.mark.parametrize("tile_m", [128, 256, "pair", "pair512"])
def test_dynamic_tile_claiming_many_tiles_per_worker(tile_m, monkeypatch):
    """Dynamic tile claiming with more than 16 tiles per worker (the in-CTA tile queue wraps around), launched
    several times in a row (the kernel re-arms its claim counters itself)."""
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import build_gemm_program, run_program

    monkeypatch.setenv("UGEMM_DYNAMIC_TILES", "1")
    torch.manual_seed(5)
    m, n, k = 8192, 24576, 128
    a = torch.randn(m, k, device=_dev()).bfloat16()
    b = (torch.randn(k, n, device=_dev()) / k ** 0.5).bfloat16()
    c = torch.zeros(m, n, device=_dev())
    prog = build_gemm_program([a], [b], c, mode=native.C_STORE, tile_m=tile_m)
    workers = prog.grid // 2 if str(tile_m).startswith("pair") else prog.grid
    assert prog.params.sched != 0 and prog.stats["tiles"] > 16 * workers
    for _ in range(3):
        run_program(prog, _dev())
    _status_ok()
    torch.testing.assert_close(c, a.float() @ b.float(), rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("method", ["stationary_b", "stationary_c"])
def test_fused_kernels_stay_inside_their_allocations(method):
    """Odd shapes on an emulated 4-rank cluster whose symmetric allocations carry guard regions: fetch warps,
    epilogue stores / red.add into 'peers' and the zeroing kernels must leave every guard byte alone."""
    m, n, k = 389, 517, 263
    full_a, full_b, full_c = make_inputs(m, n, k, seed=17, device=_dev())
    for triple in [("row", "column", "block"), ("block", "block", "block"), ("column", "row", "row")]:
        cluster = ug.EmulatedCluster(4, _dev(), guard_bytes=4096)
        mats = build_cluster_matrices(cluster, full_a, full_b, full_c, triple, 1, torch.bfloat16, torch.float32)
        run_cluster(cluster, mats, method)
        _status_ok()
        assert cluster.check_guards() == 12
        torch.testing.assert_close(mats[0][2].full_tensor().double(), oracle(full_a, full_b, full_c, torch.bfloat16),
                                   rtol=2e-3, atol=2e-3)


def test_beta_zero_with_separate_replica_reduction_clears_every_replica():
    """beta=0, Stationary-B with a column-partitioned B (no K split), replication 2 and the replica reduction as a
    separate pass: every replica fills only its share of its own copy of C, so the plan must report that all copies
    start at zero (stale rows of replica 0 would otherwise survive into the sum)."""
    from universal_gemm_b200.ops.device import DeviceState
    from universal_gemm_b200.parallel import exec as X, plan as P, runtime as R

    m, n, k = 512, 384, 320
    full_a, full_b, full_c = make_inputs(m, n, k, seed=23, device=_dev())
    cluster = ug.EmulatedCluster(4, _dev())
    mats = build_cluster_matrices(cluster, full_a, full_b, full_c * 100, ("row", "column", "row"), 2, torch.bfloat16,
                                  torch.float32)
    X.clear_program_cache()
    progs = []
    for a, b, c in mats:
        ops = P.build_stationary_b_ops(a.layout, b.layout, c.layout, rank=c.rank)
        prog, needs_zero = X._program("b", a, b, c, ops, False, 0)
        assert needs_zero
        progs.append(prog)
    st = DeviceState.get(_dev())
    for _, _, c in mats:                 # what every rank's executor does before its entry barrier
        c.local_padded.zero_()
    for prog in progs:                   # the ranks' kernels, one after the other
        prog.launch(st.stream())
    for _, _, c in mats:
        R.reduce_replicas(c)
    _status_ok()
    want = full_a.bfloat16().double() @ full_b.bfloat16().double()
    torch.testing.assert_close(mats[0][2].full_tensor(replica=0).double(), want, rtol=2e-3, atol=2e-3)
    X.clear_program_cache()
    with pytest.raises(ValueError):      # prepared plans run only the fused kernel: no separate reduction pass
        ug.prepare_matmul(*mats[0], method="stationary_b", beta=0, fuse_replica_reduce=False)


@pytest.mark.parametrize("tile_m", [128, "pair"])
@pytest.mark.parametrize("field,value", [("a_map", 4000), ("b_flag", 100000), ("seg_count", 77)])
def test_corrupt_table_entry_is_reported_not_followed(tile_m, field, value):
    """An index in the device tables that points outside the tables the launch declared (written here by the host,
    as a truncated or stale table would) is caught by the kernel's own check: it reports UG_ERR_BAD_TABLE, touches
    nothing through that index and returns; C is left alone and the next launch with intact tables works."""
    import numpy as np

    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.device import DeviceState, KernelStatusError
    from universal_gemm_b200.ops.gemm import build_gemm_program, run_program

    torch.manual_seed(3)
    m, n, k = 512, 512, 256
    a = torch.randn(m, k, device=_dev()).bfloat16()
    b = (torch.randn(k, n, device=_dev()) / k ** 0.5).bfloat16()
    c = torch.full((m, n), 5.0, device=_dev())
    prog = build_gemm_program([a], [b], c, mode=native.C_STORE, stage_b=True, tile_m=tile_m)
    tables = prog._tables
    is_task = field == "seg_count"
    dtype = native.TASK_DTYPE if is_task else native.SEGMENT_DTYPE
    off = (prog.params.tasks if is_task else prog.params.segs) - tables.data_ptr()
    good = tables[off:off + dtype.itemsize].clone()
    row = np.frombuffer(good.cpu().numpy().tobytes(), dtype=dtype).copy()
    row[0][field] = value
    tables[off:off + dtype.itemsize].copy_(torch.from_numpy(np.frombuffer(row.tobytes(), dtype=np.uint8).copy()))
    prog.params.timeout_ns = 200_000_000
    run_program(prog, _dev())
    torch.cuda.synchronize()
    with pytest.raises(KernelStatusError) as err:
        DeviceState.get(_dev()).check()
    assert err.value.code == native.ERR_BAD_TABLE
    tables[off:off + dtype.itemsize].copy_(good)
    run_program(prog, _dev())
    _status_ok()
    torch.testing.assert_close(c, a.float() @ b.float(), rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("offset,n", [(1, 1537), (2, 700), (3, 256), (1, 5), (3, 67)])
@pytest.mark.parametrize("mode", ["store", "add", "atomic"])
@pytest.mark.parametrize("tile_m", [128, 256, "pair", "pair512"])
def test_gemm_kernel_c_region_on_odd_columns(offset, n, mode, tile_m):
    """C is a column range that starts on an odd column of a wider, 16-byte-pitched matrix (what a column or block
    partition of an odd-sized C gives): the epilogue writes head columns singly and the rest as 16-byte vectors, and
    must not touch the columns next to the region."""
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import gemm

    torch.manual_seed(offset * 1000 + n)
    m, k = 300, 200
    a = torch.randn(m, k, device=_dev()).bfloat16()
    b = (torch.randn(k, n, device=_dev()) / k ** 0.5).bfloat16()
    pitch = (offset + n + 7 + 63) // 64 * 64
    big0 = torch.randn(m, pitch, device=_dev())
    big = big0.clone()
    c = big[:, offset:offset + n]
    gemm(a, b, c, mode={"store": native.C_STORE, "add": native.C_ADD, "atomic": native.C_ATOMIC}[mode], tile_m=tile_m)
    _status_ok()
    ref = a.float() @ b.float() + (0 if mode == "store" else big0[:, offset:offset + n])
    torch.testing.assert_close(c, ref, rtol=2e-3, atol=2e-3)
    assert torch.equal(big[:, :offset], big0[:, :offset]) and torch.equal(big[:, offset + n:], big0[:, offset + n:])


@pytest.mark.parametrize("method", ["stationary_c", "stationary_b"])
@pytest.mark.parametrize("triple", [("row", "column", "row"), ("column", "row", "row"), ("block", "block", "block")])
def test_skinny_problem_splits_k_across_the_gpu(method, triple):
    """M = 64 against a long K: a rank has a handful of output tiles, so the lowering cuts K into parts that add into
    C atomically (all ranks zero C first when beta = 0).  Result and beta = 1 accumulation must be unchanged."""
    from universal_gemm_b200.parallel import exec as X

    m, n, k = 64, 2100, 4500
    full_a, full_b, full_c = make_inputs(m, n, k, seed=31, device=_dev())
    cluster = ug.EmulatedCluster(8, _dev())
    mats = build_cluster_matrices(cluster, full_a, full_b, full_c, triple, 1, torch.bfloat16, torch.float32)
    X.clear_program_cache()
    prod = full_a.bfloat16().double() @ full_b.bfloat16().double()
    for _, _, c in mats:                                   # beta = 0: every rank clears its C, then all ranks add
        c.local_padded.fill_(3.0)
    progs = []
    from universal_gemm_b200.parallel import plan as P
    for a, b, c in mats:
        kind = "b" if method == "stationary_b" else "c"
        build = P.build_stationary_b_ops if kind == "b" else P.build_stationary_c_ops
        ops = build(a.layout, b.layout, c.layout, rank=c.rank)
        prog, needs_zero = X._program(kind, a, b, c, ops, True, 0)
        assert needs_zero
        progs.append((prog, c))
    assert any(p.stats["tasks"] >= 2 and p.stats["tiles"] >= 16 for p, _ in progs), [p.stats for p, _ in progs]
    if triple[0] != "column" and method == "stationary_b":   # A rows spread over the ranks and one B tile per rank:
        # the 8-row tasks of a rank share their B slices and were merged into stacked ones
        assert all(p.stats["indirect_rows"] > 0 for p, _ in progs), [p.stats for p, _ in progs]
    from universal_gemm_b200.ops.device import DeviceState
    st = DeviceState.get(_dev())
    for _, c in progs:
        c.local_padded.zero_()
    for prog, _ in progs:
        prog.launch(st.stream())
    _status_ok()
    torch.testing.assert_close(mats[0][2].full_tensor().double(), prod, rtol=2e-3, atol=2e-3)
    X.clear_program_cache()
    for a, b, c in mats:                                   # beta = 1 through the public call
        ug.matmul(a, b, c, method=method)
    _status_ok()
    torch.testing.assert_close(mats[0][2].full_tensor().double(), 2 * prod, rtol=2e-3, atol=2e-3)
    X.clear_program_cache()


@pytest.mark.parametrize("m,n,k", [(256, 512, 384), (300, 520, 200), (375, 1000, 1001), (64, 4099, 1024)])
@pytest.mark.parametrize("tile_m", [128, "pair"])
def test_gemm_kernel_fp32_operands_as_three_bf16_products(m, n, k, tile_m):
    """fp32 A and B: the fetch warps split every element into a bf16 high and low part while staging and the
    kernel accumulates lo x hi + hi x lo + hi x hi in fp32.  The result must be far closer to the fp64 product
    than a single bf16 product is (and within the reference example's tolerance for fp32 results)."""
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import gemm

    torch.manual_seed(m + k)
    a = torch.randn(m, k, device=_dev())
    b = torch.randn(k, n, device=_dev()) / k ** 0.5
    c = torch.full((m, n), 9.0, device=_dev())
    gemm(a, b, c, mode=native.C_STORE, tile_m=tile_m)
    _status_ok()
    want = a.double() @ b.double()
    err = (c.double() - want).abs().max().item()
    bf16_err = ((a.bfloat16().double() @ b.bfloat16().double()) - want).abs().max().item()
    assert err < 1e-4 and err < bf16_err / 50, (err, bf16_err)


@pytest.mark.parametrize("method", ["stationary_c", "stationary_b"])
def test_fused_fp32_operands_emulated(method):
    m, n, k = 301, 203, 517
    full_a, full_b, full_c = make_inputs(m, n, k, seed=41, device=_dev())
    for triple in [("row", "column", "row"), ("block", "block", "block"), ("column", "row", "row")]:
        cluster = ug.EmulatedCluster(4, _dev(), guard_bytes=4096)
        mats = build_cluster_matrices(cluster, full_a, full_b, full_c, triple, 1, torch.float32, torch.float32)
        run_cluster(cluster, mats, method)
        _status_ok()
        assert cluster.check_guards() == 12
        want = full_c.double() + full_a.double() @ full_b.double()
        torch.testing.assert_close(mats[0][2].full_tensor().double(), want, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("m,n,k,tile_m", [(3001, 3001, 3001, "pair"), (3001, 3001, 3001, 256), (12289, 1537, 3001, 128),
                                          (64, 16383, 16383, None), (1537, 12289, 12289, "pair512")])
def test_gemm_kernel_large_odd_shapes(m, n, k, tile_m):
    """Odd sizes of the benchmark sweep at kernel level: odd pitches put A and B on the 2-byte gather path of the
    fetch warps, C is written with ragged right and bottom edges, M = 64 leaves most tensor rows empty."""
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import gemm

    torch.manual_seed(m + n)
    a = torch.randn(m, k, device=_dev()).bfloat16()
    b = (torch.randn(k, n, device=_dev()) / k ** 0.5).bfloat16()
    c = torch.full((m, n), 2.0, device=_dev())
    gemm(a, b, c, mode=native.C_ADD, tile_m=tile_m)
    _status_ok()
    torch.testing.assert_close(c, a.float() @ b.float() + 2.0, rtol=3e-3, atol=3e-3)


@pytest.mark.parametrize("case", ["aligned", "odd", "skinny", "bf16_c", "replicated"])
def test_epilogue_checksum_adds_up_to_the_sum_of_the_product(case):
    """``checksum=``: every rank's kernel adds the sum of all values it writes into (or adds to) C to a running
    double; over all ranks that is sum(A @ B), whatever path the epilogue takes (vector, shifted for odd columns,
    row table of merged skinny tasks with K split, bf16 output, pushes into replica 0) and over repeated calls."""
    m, n, k, triple, rep, c_dtype, world = {
        "aligned": (1024, 1536, 512, ("row", "column", "row"), 1, torch.float32, 4),
        "odd": (389, 517, 263, ("block", "column", "block"), 1, torch.float32, 4),
        "skinny": (64, 2100, 4500, ("row", "column", "row"), 1, torch.float32, 8),
        "bf16_c": (512, 777, 320, ("column", "row", "row"), 1, torch.bfloat16, 4),
        "replicated": (512, 768, 640, ("row", "row", "row"), 2, torch.float32, 4),
    }[case]
    full_a, full_b, full_c = make_inputs(m, n, k, seed=51, device=_dev())
    want = float((full_a.bfloat16().double() @ full_b.bfloat16().double()).sum().item())
    scale = float((full_a.bfloat16().double() @ full_b.bfloat16().double()).abs().sum().item())
    for method in ("stationary_c", "stationary_b"):
        cluster = ug.EmulatedCluster(world, _dev())
        mats = build_cluster_matrices(cluster, full_a, full_b, full_c, triple, rep, torch.bfloat16, c_dtype)
        sums = [torch.zeros(1, dtype=torch.float64, device=_dev()) for _ in mats]
        calls = 2
        for _ in range(calls):
            for (a, b, c), chk in zip(mats, sums):
                ug.matmul(a, b, c, method=method, checksum=chk)
        _status_ok()
        got = sum(float(x.item()) for x in sums)
        assert abs(got - calls * want) <= 1e-5 * scale + 1e-6, (case, method, got, calls * want)


@pytest.mark.parametrize("src_dtype,dst_dtype", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32),
                                                 (torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_move_pieces_every_shape_and_phase(src_dtype, dst_dtype):
    """Batched copy / conversion: vectors in and out of phase, single elements (odd pitches), rows from one element to
    several jobs, more pieces than one launch takes.  Exact (copies, and one rounding to nearest), and nothing outside the pieces is written."""
    import numpy as np

    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.device import DeviceState

    st = DeviceState.get(_dev())
    gen = torch.Generator(device=_dev()).manual_seed(5)
    code = {torch.float32: native.DT_F32, torch.bfloat16: native.DT_BF16}
    shapes = [(r, c) for r in (1, 5, 17) for c in (1, 31, 33, 127, 130, 255, 256, 512, 515, 1024, 2048, 2053)]
    for s_off, d_off, s_ld, d_ld in ((0, 0, 2112, 2176), (3, 0, 2112, 2176), (0, 5, 2112, 2176), (8, 8, 2109, 2175)):
        pieces = np.zeros(len(shapes) * 2, dtype=native.MOVE_PIECE_DTYPE)
        rows_total = 2 * sum(r + 1 for r, _ in shapes)
        src = torch.randn(rows_total, s_ld, device=_dev(), generator=gen).to(src_dtype)
        src[0, :4] = torch.tensor([float("inf"), float("-inf"), float("nan"), -0.0], device=_dev()).to(src_dtype)
        dst = torch.full((rows_total, d_ld), 7.0, device=_dev(), dtype=dst_dtype)
        want = dst.clone()
        row = 0
        for i, (r, c) in enumerate(shapes + shapes):
            sv, dv = src[row:row + r, s_off:s_off + c], dst[row:row + r, d_off:d_off + c]
            pieces[i] = (dv.data_ptr(), sv.data_ptr(), c, r, 0)
            want[row:row + r, d_off:d_off + c] = sv.to(dst_dtype)
            row += r + 1
        st.move_pieces(pieces, d_ld, code[dst_dtype], s_ld, code[src_dtype])
        torch.cuda.synchronize()
        bits = torch.int32 if dst_dtype == torch.float32 else torch.int16
        assert torch.equal(dst.isnan(), want.isnan())
        assert torch.equal(dst.nan_to_num(nan=1.0).view(bits), want.nan_to_num(nan=1.0).view(bits))


@pytest.mark.parametrize("src_part,dst_part", [("row", "column"), ("column", "block"), ("block", "row")])
@pytest.mark.parametrize("src_dtype,dst_dtype", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32),
                                                 (torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16),
                                                 (torch.int32, torch.int32)])
def test_redistribute_converts_on_the_way(src_part, dst_part, src_dtype, dst_dtype):
    """Against the tensor path of a CPU cluster; empty trailing tiles (5 rows on 8 ranks) among the sizes."""
    for rows, cols, world in ((301, 203, 4), (5, 1037, 8), (640, 512, 8)):
        full = (torch.randn(rows, cols) * 50).to(src_dtype)
        got, want = [], []
        for dev, keep in ((_dev(), got), (torch.device("cpu"), want)):
            srcs = [ug.distribute_tensor(full.to(dev), w, src_part, dtype=src_dtype)
                    for w in ug.EmulatedCluster(world, dev).worlds()]
            keep += [ug.redistribute(s, dst_part, dtype=dst_dtype).local.cpu() for s in srcs]
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert torch.equal(g, w)


@pytest.mark.parametrize("m,n,k", [(256, 512, 128), (300, 1000, 200), (375, 1537, 1001), (64, 2100, 1984), (1, 33, 64)])
@pytest.mark.parametrize("tile_m", [128, 256, "pair", "pair512"])
def test_gelu_from_the_epilogue(m, n, k, tile_m, monkeypatch):
    """C and gelu(C) of one launch: C equals the plain product (up to the order of its fp32 sums), the activation is the exact gelu of that C
    up to one bf16 rounding (2^-8 relative, and fp32 error of the distribution function near zero), padding untouched."""
    from universal_gemm_b200.parallel import exec as X

    monkeypatch.setenv("UGEMM_TILE_M", str(tile_m))
    full_a, full_b, _ = make_inputs(m, n, k, seed=41, device=_dev())
    world = ug.SingleWorld(_dev())
    a = ug.distribute_tensor(full_a, world, "row", dtype=torch.bfloat16)
    b = ug.distribute_tensor(full_b, world, "column", dtype=torch.bfloat16)
    c, plain = ug.zeros(world, (m, n), "row", torch.float32), ug.zeros(world, (m, n), "row", torch.float32)
    act = ug.zeros(world, (m, n), "row", torch.bfloat16)
    act.local_padded.fill_(7.0)
    X.clear_program_cache()
    assert X.can_fuse_gelu("c", a, b, c, act)
    X.matmul_gelu(a, b, c, act, method="stationary_c")
    ug.matmul(a, b, plain, method="stationary_c", beta=0)
    _status_ok()
    torch.testing.assert_close(c.local, plain.local, rtol=1e-5, atol=1e-5)
    want = torch.nn.functional.gelu(c.local.double())
    assert ((act.local.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()
    assert (act.local_padded[:, n:] == 7.0).all()
    X.clear_program_cache()


@pytest.mark.parametrize("method,triple", [("stationary_c", ("row", "column", "row")), ("stationary_b", ("row", "column", "row")),
                                           ("stationary_c", ("block", "row", "block"))])
def test_matmul_gelu_on_several_ranks(method, triple):
    """Stationary-C writes the activation from the epilogue; Stationary-B, whose peers store into C, takes the pass."""
    from universal_gemm_b200.parallel import exec as X

    m, n, k = 515, 1030, 300
    full_a, full_b, _ = make_inputs(m, n, k, seed=42, device=_dev())
    mats = []
    for w in ug.EmulatedCluster(4, _dev()).worlds():
        mats.append((ug.distribute_tensor(full_a, w, triple[0], dtype=torch.bfloat16),
                     ug.distribute_tensor(full_b, w, triple[1], dtype=torch.bfloat16),
                     ug.zeros(w, (m, n), triple[2], torch.float32), ug.zeros(w, (m, n), triple[2], torch.bfloat16)))
    X.clear_program_cache()
    for _ in range(2):          # emulated ranks run one after the other: in the second round all peers have stored
        for a, b, c, act in mats:
            assert X.can_fuse_gelu(method[-1], a, b, c, act) == (method == "stationary_c")
            X.matmul_gelu(a, b, c, act, method=method)
    _status_ok()
    want = torch.nn.functional.gelu(full_a.bfloat16().double() @ full_b.bfloat16().double())
    torch.testing.assert_close(mats[0][3].full_tensor().double(), want, rtol=1e-2, atol=4e-3)
    X.clear_program_cache()


def test_counters_are_back_at_zero_after_a_launch():
    """Programs that stage operands run many times without a clearing pass."""
    from universal_gemm_b200.parallel import exec as X

    m, n, k = 515, 700, 2100
    full_a, full_b, _ = make_inputs(m, n, k, seed=43, device=_dev())
    cluster = ug.EmulatedCluster(2, _dev())
    mats = build_cluster_matrices(cluster, full_a, full_b, torch.zeros(m, n, device=_dev()), ("block", "row", "column"), 1,
                                  torch.bfloat16, torch.float32)
    X.clear_program_cache()
    want = full_a.bfloat16().double() @ full_b.bfloat16().double()
    for _ in range(3):
        for a, b, c in mats:
            c.local_padded.fill_(9.0)
            ug.matmul(a, b, c, method="stationary_c", beta=0)
    for label, prog in X.cached_programs():
        assert prog.params.num_pieces > 0 and prog.params.finished != 0
        at = prog.params.flags - prog._tables.data_ptr()
        words = prog._tables[at:at + 4 * (prog.params.num_flags + 2)].view(torch.int32)
        assert int(words.abs().sum()) == 0, label
        for at in (prog.params.sched, prog.params.finished):          # the next claim of a tile, the workers that are done
            if at:
                at -= prog._tables.data_ptr()
                assert int(prog._tables[at:at + 4].view(torch.int32)) == 0, label
    _status_ok()
    torch.testing.assert_close(mats[0][2].full_tensor().double(), want, rtol=2e-3, atol=2e-3)
    X.clear_program_cache()


def _cut_program(a, b, c, mode, tile_m, parts, **operand):
    from universal_gemm_b200.ops.device import DeviceState, torch_dtype_code
    from universal_gemm_b200.ops.fused import FusedProgramBuilder, TaskSpec
    from universal_gemm_b200.ops.gemm import _segments, _slice_of

    st = DeviceState.get(_dev())
    builder = FusedProgramBuilder(_dev(), num_sms=st.num_sms, tile_m=tile_m, parts=parts)
    builder.add_task(TaskSpec(c_ptr=c.data_ptr(), ldc=c.stride(0), m=a.shape[0], n=b.shape[1], c_mode=mode,
                              c_dtype=torch_dtype_code(c.dtype), segments=_segments(_slice_of(a, **operand), _slice_of(b, **operand))))
    return builder.build(st.status_ptr)


@pytest.mark.parametrize("m,n,k,parts", [(128, 256, 128, 2), (300, 520, 712, 3), (257, 1029, 1000, 5), (64, 2049, 4160, 8),
                                         (1, 3, 640, 2)])
@pytest.mark.parametrize("mode,c_dtype", [("store", torch.float32), ("add", torch.float32), ("atomic", torch.float32),
                                          ("store", torch.bfloat16), ("add", torch.bfloat16)])
@pytest.mark.parametrize("tile_m", [128, 256, "pair"])
def test_cut_tiles_sum_their_parts(m, n, k, parts, mode, c_dtype, tile_m):
    """Every tile cut into K parts (uneven shares, ragged K, odd columns): one result per element, whoever writes it,
    as accurate as an uncut tile; the same bits on every launch, and the counters are back at zero."""
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import run_program

    gen = torch.Generator(device=_dev()).manual_seed(7)
    a = torch.randn(m, k + (-k) % 8, device=_dev(), generator=gen).bfloat16()[:, :k]
    b = (torch.randn(k, n, device=_dev(), generator=gen) / k ** 0.5).bfloat16()
    prod = a.double() @ b.double()
    code = {"store": native.C_STORE, "add": native.C_ADD, "atomic": native.C_ATOMIC}[mode]
    for offset in (0, 1):                                 # C on a 16-byte boundary, and on an odd column
        wide = torch.full((m, n + 8), 2.0, device=_dev(), dtype=c_dtype)
        c = wide[:, offset:offset + n]
        prog = _cut_program(a, b, c, code, tile_m, parts)
        assert prog.stats["parts"] == parts and prog.stats["cut_tiles"] > 0
        seen = []
        for _ in range(2):
            wide.fill_(2.0)
            run_program(prog, _dev())
            seen.append(c.clone())
        _status_ok()
        want = prod + (0.0 if mode == "store" else 2.0)
        # fp32: the sums' own error.  bf16 (8 significant bits): half an ulp (2^-8 relative) for the sum taken from the accumulator and, when it
        # is added to C, another one for the result.
        bound = 1e-5 * want.abs() if c_dtype == torch.float32 else 1.01 * 2.0 ** -8 * (prod.abs() + want.abs())
        assert ((seen[0].double() - want).abs() <= bound + 2e-5).all()
        assert torch.equal(seen[0], seen[1])
        assert (wide[:, :offset] == 2.0).all() and (wide[:, offset + n:] == 2.0).all()
        at = prog.params.part_flags - prog._tables.data_ptr()
        assert int(prog._tables[at:at + 4 * prog.params.num_part_flags].view(torch.int32).abs().sum()) == 0


@pytest.mark.parametrize("tile_m", [128, 256, "pair"])
def test_cut_tiles_with_staged_operands_and_fp32_split(tile_m):
    """The parts of a tile share its staged copies (K ranges, small terms first)."""
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import run_program

    gen = torch.Generator(device=_dev()).manual_seed(8)
    m, n, k = 300, 700, 2200
    for dtype, tol in ((torch.bfloat16, 1e-5), (torch.float32, 3e-5)):
        a = torch.randn(m, k, device=_dev(), generator=gen).to(dtype)
        b = (torch.randn(k, n, device=_dev(), generator=gen) / k ** 0.5).to(dtype)
        c = torch.zeros(m, n, device=_dev())
        prog = _cut_program(a, b, c, native.C_STORE, tile_m, 4, remote=True)
        for _ in range(2):
            run_program(prog, _dev())
        _status_ok()
        want = a.double() @ b.double()
        assert (c.double() - want).norm() <= tol * want.norm()


@pytest.mark.parametrize("tile_m", [128, 256, "pair", "pair512"])
@pytest.mark.parametrize("n", [64, 65, 255, 256, 449, 1030])
def test_one_load_for_all_column_chunks_of_b(tile_m, n, monkeypatch):
    """B read in place, all 64-column chunks of a tile by one load: the last chunk of a ragged width reads the padding of
    the rows (NaN here), which must not reach any element of C."""
    from universal_gemm_b200.parallel import exec as X

    monkeypatch.setenv("UGEMM_TILE_M", str(tile_m))
    m, k = 200, 328
    full_a, full_b, _ = make_inputs(m, n, k, seed=44, device=_dev())
    world = ug.SingleWorld(_dev())
    a = ug.distribute_tensor(full_a, world, "row", dtype=torch.bfloat16)
    b = ug.distribute_tensor(full_b, world, "column", dtype=torch.bfloat16)
    b.local_padded[:, n:] = float("nan")
    c = ug.zeros(world, (m, n), "row", torch.float32)
    X.clear_program_cache()
    ug.matmul(a, b, c, method="stationary_c", beta=0)
    _status_ok()
    want = full_a.bfloat16().double() @ full_b.bfloat16().double()
    torch.testing.assert_close(c.local.double(), want, rtol=2e-3, atol=2e-3)
    X.clear_program_cache()


@pytest.mark.parametrize("m,n,k", [(200, 300, 2500), (64, 1030, 4097), (515, 700, 2048)])
@pytest.mark.parametrize("beta", [0, 1])
def test_small_fp32_products_share_their_staged_copies(m, n, k, beta):
    """Few tiles, long K, fp32 operands: the parts are ranges of K blocks over one staged copy of each operand."""
    from universal_gemm_b200.parallel import exec as X

    full_a, full_b, full_c = make_inputs(m, n, k, seed=45, device=_dev())
    world = ug.SingleWorld(_dev())
    a = ug.distribute_tensor(full_a, world, "row", dtype=torch.float32)
    b = ug.distribute_tensor(full_b, world, "row", dtype=torch.float32)
    c = ug.distribute_tensor(full_c, world, "row", dtype=torch.float32)
    X.clear_program_cache()
    ug.matmul(a, b, c, beta=beta)
    _status_ok()
    (_, prog), = X.cached_programs()
    staged = 4 * 2 * (m * (-(-k // 64) * 64) + k * (-(-n // 64) * 64)) // 2 + 4 * 1024
    assert prog.stats["tasks"] > 1 and prog.stats["staged_bytes"] <= staged, prog.stats
    want = full_a.double() @ full_b.double() + beta * full_c.double()
    assert (c.local.double() - want).norm() <= 3e-5 * want.norm()
    X.clear_program_cache()


@pytest.mark.parametrize("tile_m", [128, 256, "pair"])
def test_the_last_part_of_a_tile_sees_all_other_parts(tile_m):
    """Every lane of the part that writes C reads what other SMs have just written: 100 launches over changing operands,
    so that a sum of the launch before would show, each equal in every bit to a second launch on the same operands."""
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import run_program

    m, n, k = 256, 1024, 2048
    gen = torch.Generator(device=_dev()).manual_seed(9)
    source = torch.randn(m, k, device=_dev(), generator=gen).bfloat16()
    a = source.clone()
    b = (torch.randn(k, n, device=_dev(), generator=gen) / k ** 0.5).bfloat16()
    c = torch.zeros(m, n, device=_dev())
    prog = _cut_program(a, b, c, native.C_STORE, tile_m, 8)
    differ = torch.zeros((), dtype=torch.int64, device=_dev())
    for i in range(50):
        a.copy_(source.roll(i, 0))
        run_program(prog, _dev())
        first = c.clone()
        if i == 0:
            base = first
        run_program(prog, _dev())
        differ += (first != c).sum() + (first != base.roll(i, 0)).sum()
    _status_ok()
    assert int(differ) == 0
    want = source.double() @ b.double()
    assert (base.double() - want).norm() <= 1e-5 * want.norm()


@pytest.mark.parametrize("n", [1, 31, 33, 95, 97, 255, 279, 543])
@pytest.mark.parametrize("tile_m", [128, 256, "pair"])
def test_bf16_add_rounds_once_at_the_ragged_end(n, tile_m):
    """bf16 ``C +=`` onto values that nearly cancel the product, in a C with aligned rows: the columns past the last whole
    chunk of 32 add the fp32 sum and round once, so what is left is within half an ulp (2^-9 relative) of the exact value,
    plus the error of an fp32 sum of k products (k 2^-24 of the sum of their sizes: 1.5e-4 here).  Rounding the product
    first leaves up to 2^-9 of the product, 1e-3 and more."""
    from universal_gemm_b200.ops import native
    from universal_gemm_b200.ops.gemm import build_gemm_program, run_program

    m, k = 200, 256
    gen = torch.Generator(device=_dev()).manual_seed(10 + n)
    a = torch.randn(m, k, device=_dev(), generator=gen).bfloat16()
    b = torch.zeros(k, -(-n // 64) * 64, device=_dev(), dtype=torch.bfloat16)[:, :n]
    b.copy_(torch.randn(k, n, device=_dev(), generator=gen) / k ** 0.5)
    c = torch.zeros(m, -(-n // 64) * 64, device=_dev(), dtype=torch.bfloat16)[:, :n]
    prod = a.double() @ b.double()
    sums = k * 2.0 ** -24 * (a.double().abs() @ b.double().abs())
    c.copy_(-prod)                                             # rounded to bf16: the sum is that rounding's error
    want = prod + c.double()
    run_program(build_gemm_program([a], [b], c, mode=native.C_ADD, tile_m=tile_m), _dev())
    _status_ok()
    # the two warps of a lane quadrant split a tile's columns at a multiple of 64, so chunks of 32 start at multiples of 32
    ragged = n // 32 * 32
    got, left = c[:, ragged:].double(), want[:, ragged:]
    assert ((got - left).abs() <= 1.01 * 2.0 ** -9 * left.abs() + sums[:, ragged:]).all()
    whole, prod = (c.double() - want)[:, :ragged].abs(), prod[:, :ragged].abs()
    assert (whole <= 1.01 * 2.0 ** -9 * (2 * prod + want[:, :ragged].abs()) + sums[:, :ragged]).all()
