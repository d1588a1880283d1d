"""How long a lowered program lives and which call it serves.  The lowering itself is replaced (it needs a GPU): what is
tested is the cache, on matrices of CPU clusters whose buffers are told which addresses they have."""
import gc
import weakref

import pytest
import torch

import universal_gemm_b200 as ug
from universal_gemm_b200.parallel import exec as X
from universal_gemm_b200.parallel import plan as P
from universal_gemm_b200.parallel import prepared


class _Program:
    def __init__(self, addresses, dtypes):
        self.addresses, self.dtypes, self.launched = addresses, dtypes, 0


@pytest.fixture(autouse=True)
def lowered(monkeypatch):
    """Every lowering, as (addresses of all ranks' tiles, dtypes) of A, B, C."""
    seen = []

    def lower(kind, a, b, c, ops, **options):
        mats = [m for m in (a, b, c, options.get("gelu_out")) if m is not None]
        seen.append(weakref.ref(prog := _Program([list(m.buffer._ptrs) for m in mats], [m.dtype for m in mats])))
        return prog, False

    monkeypatch.setattr(X, "lower_plan", lower)
    X.clear_program_cache()
    yield seen
    X.clear_program_cache()


def _triple(ptrs, dtype=torch.bfloat16, c_dtype=torch.float32, world=2):
    """A, B, C of rank 0, with the given addresses of (rank 0's, rank 1's) tiles."""
    worlds = ug.EmulatedCluster(world, "cpu").worlds()
    mats = [(ug.empty(w, (64, 64), "row", dtype), ug.empty(w, (64, 64), "column", dtype), ug.empty(w, (64, 64), "row", c_dtype))
            for w in worlds]
    for i, m in enumerate(mats[0]):
        m.buffer._ptrs = [p + 65536 * i for p in ptrs]
    return mats[0]


def _get(a, b, c, kind="c", ops=None, **kw):
    build = P.build_stationary_c_ops if kind == "c" else P.build_stationary_b_ops
    return X._program(kind, a, b, c, build(a.layout, b.layout, c.layout, rank=0) if ops is None else ops, True, **kw)[0]


def test_a_program_serves_its_own_matrices_again():
    a, b, c = _triple([1 << 20, 2 << 20])
    prog = _get(a, b, c)
    assert _get(a, b, c) is prog and _get(a, b, c, beta=0) is not prog and _get(a, b, c) is prog
    assert [p for _, p in X.cached_programs()][0] is prog


def test_own_addresses_that_come_back_with_other_peers_are_lowered_again():
    """Rank 0's tiles get their old addresses, rank 1's do not: the old program would fetch from and push to memory that
    rank 1 no longer has."""
    first = _triple([1 << 20, 2 << 20])
    old = _get(*first)
    second = _triple([1 << 20, 5 << 20])
    new = _get(*second)
    assert new is not old and new.addresses[0] == [1 << 20, 5 << 20]
    assert _get(*first) is old


@pytest.mark.parametrize("then", [dict(c_dtype=torch.bfloat16), dict(dtype=torch.float32)])
def test_an_address_that_comes_back_with_another_dtype_is_lowered_again(then):
    """Half (or twice) the bytes lie at the same address: the old program would write or read past the end."""
    old = _get(*_triple([1 << 20, 2 << 20]))
    mats = _triple([1 << 20, 2 << 20], **then)
    new = _get(*mats)
    assert new is not old and new.dtypes == [m.dtype for m in mats]


@pytest.mark.parametrize("which", [0, 1, 2, 3])
def test_a_program_goes_with_the_first_of_its_matrices(which, lowered):
    """Collected (nothing calls free() then): the program, its tables and its workspace are given back."""
    mats = list(_triple([1 << 20, 2 << 20])) + [ug.empty(ug.SingleWorld("cpu"), (64, 64), "row", torch.bfloat16)]
    _get(*mats[:3], gelu_out=mats[3])
    other = _triple([3 << 20, 4 << 20])
    keep = _get(*other)
    gc.collect()
    assert lowered[0]() is not None and len(X._program_cache) == 2
    del mats[which]
    gc.collect()
    assert lowered[0]() is None and len(X._program_cache) == 1
    assert _get(*other) is keep


def test_a_weight_remembers_only_the_programs_that_are_left():
    """A loop over new inputs and results with one weight: nothing of the earlier calls stays."""
    a, b, c = _triple([1 << 20, 2 << 20])
    _get(a, b, c)
    for i in range(5):
        x, _, y = _triple([(3 + i) << 20, 2 << 20])
        _get(x, b, y)
        del x, y
        gc.collect()
        assert len(X._program_cache) == 1 and len(X._programs_of[b.buffer.uid]) == 1


def test_freeing_a_matrix_drops_its_programs_only():
    a, b, c = _triple([1 << 20, 2 << 20])
    other = _triple([3 << 20, 4 << 20])
    _get(a, b, c), _get(a, b, other[2])
    keep = _get(*other)
    c.free()
    assert len(X._program_cache) == 2
    b.free()
    assert len(X._program_cache) == 1 and _get(*other) is keep


def test_op_lists_of_the_same_matrices_do_not_replace_each_other(lowered):
    """A launch (or a graph) of the one may be in flight when the other is lowered."""
    a, b, c = _triple([1 << 20, 2 << 20])
    ops = P.build_stationary_c_ops(a.layout, b.layout, c.layout, rank=0)
    whole, part = _get(a, b, c, ops=ops), _get(a, b, c, ops=ops[:1])
    assert whole is not part
    assert _get(a, b, c, ops=list(ops)) is whole and _get(a, b, c, ops=list(ops[:1])) is part
    for i in range(3 * X._MAX_OP_LISTS):                       # bounded all the same
        _get(a, b, c, ops=[ops[0]] * (i + 2))
    assert len(X._program_cache) == X._MAX_OP_LISTS
    assert _get(a, b, c, ops=ops) is whole


def test_a_prepared_plan_keeps_its_program(monkeypatch, lowered):
    """Its graph holds the addresses of the program's tables: neither clearing the cache nor other plans may free them."""
    monkeypatch.setattr(X, "_can_fuse", lambda *mats: True)
    ran = []
    monkeypatch.setattr(X, "_run_fused", lambda *args, program=None, **kw: ran.append(program))
    a, b, c = _triple([1 << 20, 2 << 20])
    plan = prepared.prepare_matmul(a, b, c)
    X.clear_program_cache()
    gc.collect()
    plan()
    assert len(lowered) == 1 and ran == [(lowered[0](), False)] and ran[0][0] is plan.program
