"""Several steps of a batch per launch against one step per launch, bit for bit:
uneven instances (narrow and wide, whole vectors and odd rows, the smallest
that each form takes), every boundary, retired instances, graph capture; and
the plan's own limits."""

import numpy as np
import pytest
import torch

from latticeboltzmann_gb300 import _lib
from latticeboltzmann_gb300 import batch as B

pytestmark = pytest.mark.gpu

SINGLE = {"flat": True, "vector": False, "rows": 1, "threads": 256, "blocks": 608}
SMALL = [(2, 2), (5, 3), (16, 16), (17, 40), (64, 33), (40, 130), (9, 300), (300, 9)]
# more than 1.2 M cells: the march (groups of 8, 16 and 32 lanes, odd and even rows, chunks past the end)
LARGE = [(8, 16), (9, 17), (11, 24), (40, 25), (33, 56), (50, 57), (21, 120), (70, 121), (100, 144), (130, 145),
         (1100, 511), (1024, 512), (300, 333)]


def make(sizes, storage, boundary, cuda, seed=3):
    om = np.linspace(0.7, 1.8, len(sizes))
    b = B.BatchedLattice(sizes, om, boundary=boundary, u0=np.linspace(0.03, 0.1, len(sizes)), storage=storage,
                         device=cuda)
    g = torch.Generator(device=cuda).manual_seed(seed)

    def fields(i):
        r = [torch.randn(*sizes[i], generator=g, dtype=torch.float64, device=cuda) for _ in range(3)]
        return 1 + 0.02 * r[0], 0.03 * r[1], 0.03 * r[2]
    return b.equilibrium(fields)


def same(sizes, storage, boundary, cuda, kind, parts):
    a, b = make(sizes, storage, boundary, cuda), make(sizes, storage, boundary, cuda)
    assert a._several()[0] == kind
    for n in parts:
        a.step(n)
        b.step(n, SINGLE)
    assert torch.equal(a.state, b.state)
    return a, b


@pytest.mark.parametrize("storage", ["f32", "f32dev", "f64", "f16dev", "bf16dev"])
@pytest.mark.parametrize("boundary", ["periodic", "cavity", "cavity-ladd"])
def test_small_batches(cuda, storage, boundary):
    same(SMALL, storage, boundary, cuda, _lib.BATCH_TILE, (1, 2, 13))
    same([(96, 96)] * 3, storage, boundary, cuda, _lib.BATCH_TILE, (8, 5))
    same([(200, 210)], storage, boundary, cuda, _lib.BATCH_TILE, (20,))


@pytest.mark.parametrize("storage", ["f32", "f32dev"])
@pytest.mark.parametrize("boundary", ["periodic", "cavity", "cavity-ladd"])
def test_large_batches(cuda, storage, boundary):
    same(LARGE, storage, boundary, cuda, _lib.BATCH_MARCH, (4, 2, 7))


@pytest.mark.parametrize("sizes", [SMALL, LARGE])
def test_retired_instances_keep_their_state(cuda, sizes):
    a, b = same(sizes, "f32", "cavity", cuda, _lib.BATCH_TILE if sizes is SMALL else _lib.BATCH_MARCH, (6,))
    mask = np.arange(len(sizes)) % 3 != 1
    frozen = {i: a.populations(i) for i in np.nonzero(~mask)[0]}
    a.set_active(mask)
    b.set_active(mask)
    a.step(11)
    b.step(11, SINGLE)
    for i in range(len(sizes)):
        assert torch.equal(a.populations(i), b.populations(i))
    for i, f in frozen.items():
        assert torch.equal(a.populations(i), f)
    a.set_active(np.zeros(len(sizes), dtype=bool))
    before = a.state.clone()
    a.step(5)
    for i in range(len(sizes)):
        nx, ny = sizes[i]
        off = int(a._table_np["offset"][i])
        assert torch.equal(a.state[off:off + 9 * nx * ny], before[off:off + 9 * nx * ny])


@pytest.mark.parametrize("sizes", [SMALL, LARGE])
def test_capture(cuda, sizes):
    for n in (2, 6, 10, 12):
        a, b = make(sizes, "f32", "periodic", cuda), make(sizes, "f32", "periodic", cuda)
        replay = a.capture(n)
        replay()
        replay()
        b.step(2 * n, SINGLE)
        assert torch.equal(a.state, b.state)


def test_single_steps_where_several_do_not_apply(cuda):
    assert make([(1, 9), (4, 4)], "f32", "periodic", cuda)._several()[0] == _lib.BATCH_SINGLE
    assert B.BatchedLattice([(2000, 800)], [1.0], storage="f64", device=cuda)._several()[0] == _lib.BATCH_SINGLE
    assert B.BatchedLattice([(2000, 800), (7, 40)], [1.0, 1.0], device=cuda)._several()[0] == _lib.BATCH_SINGLE
    saved = _lib.get_tuning(_lib.TUNE_TWO_STEP)
    try:
        _lib.set_tuning(_lib.TUNE_TWO_STEP, 0)
        assert make([(8, 16)], "f32", "periodic", cuda)._several()[0] == _lib.BATCH_SINGLE
    finally:
        _lib.set_tuning(_lib.TUNE_TWO_STEP, saved)


def test_tasks_that_do_not_fit_are_skipped(cuda):
    """A task of another batch's shape (rows or columns past the instance, an
    instance that is not there) changes nothing."""
    a = make([(16, 32), (24, 40)], "f32", "periodic", cuda)
    kind = _lib.BATCH_TILE
    bad = torch.tensor([[2, 0, 0, 4 | 4 << 16], [-1, 0, 0, 4 | 4 << 16], [0, 14, 0, 4 | 4 << 16], [0, 0, 30, 4 | 4 << 16],
                        [1, -1, 0, 4 | 4 << 16], [0, 0, 0, 0]], dtype=torch.int32, device=cuda)
    dst = torch.zeros_like(a.state)
    _lib.call("lbgb_batch_steps", a.state.data_ptr(), dst.data_ptr(), a.total, a._table(True).data_ptr(), a.n,
              bad.data_ptr(), len(bad), kind, 3, a.bcode, a.code, torch.cuda.current_stream(cuda).cuda_stream)
    march = torch.tensor([[2, 0, 0, 4 | 32 << 16], [0, 16, 0, 4 | 32 << 16], [0, 0, 32, 4 | 32 << 16],
                          [0, 0, 0, 13 | 32 << 16], [0, 0, 0, 4 | 12 << 16], [0, 0, 0, 32 << 16]], dtype=torch.int32,
                         device=cuda)
    _lib.call("lbgb_batch_steps", a.state.data_ptr(), dst.data_ptr(), a.total, a._table(True).data_ptr(), a.n,
              march.data_ptr(), len(march), _lib.BATCH_MARCH, 4, a.bcode, a.code,
              torch.cuda.current_stream(cuda).cuda_stream)
    torch.cuda.synchronize()
    assert float(dst.abs().max()) == 0.0
