"""Edges of the kernels' tiles, work splits and dispatch rules, against float64 products of the
bit-exactly dequantized weights (or the CPU oracle where the dequantization is not the point)."""
import numpy as np
import pytest
import torch

from gufo_npu_b200 import quantize as Q
from gufo_npu_b200.backend import Context
from tests.golden import make_golden as G

pytestmark = pytest.mark.gpu


def rel_l2(got, want):
    got = np.asarray(got, dtype=np.float64).ravel()
    want = np.asarray(want, dtype=np.float64).ravel()
    return float(np.linalg.norm(got - want) / max(np.linalg.norm(want), 1e-30))


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def _matrix(ctx, ggml_type, rows, cols, seed):
    """A matrix handle and its values in float64."""
    raw = Q.quantize(ggml_type, torch.from_numpy(G.normal(seed, rows, cols) * 0.02)).numpy().reshape(rows, -1)
    m = ctx.matrix_upload(ggml_type, raw, rows, cols)
    return m, ctx.dequantize(m, 0, rows, cols).astype(np.float64)


@pytest.mark.parametrize("ggml_type", [Q.GGML_Q4_K, Q.GGML_Q6_K])
@pytest.mark.parametrize("tokens,rows,cols", [
    (17, 1, 256),        # one row of a 128-row tile, one step
    (32, 127, 2304),     # nine blocks: a Q6_K slab of one
    (192, 129, 512),     # the widest token group; a tile of one row
    (193, 300, 512),     # two groups, the second nearly empty
    (513, 257, 768),     # three groups
    (40, 2560, 1024),    # few tiles: every one shared by several thread blocks
    (24, 19000, 512),    # 149 tiles: cuts through most of them
])
def test_gemm_tiles_groups_and_cuts(ctx, ggml_type, tokens, rows, cols):
    m, w = _matrix(ctx, ggml_type, rows, cols, 70 + rows % 11)
    x = G.normal(80 + tokens, tokens, cols)
    want = x.astype(np.float64) @ w.T
    for _ in range(2):   # the second run meets the counters the first has left
        got = ctx.matmul([(m, 0, rows)], x, tokens, rows)
        ctx.synchronize()
        assert rel_l2(got, want) <= 5e-4
        for t in range(tokens if rows > 100 else 0):
            assert rel_l2(got[t], want[t]) <= 1e-3, t
    ctx.matrix_free(m)


@pytest.mark.parametrize("tokens", [1, 2, 3, 8, 9, 33])
@pytest.mark.parametrize("rows,cols", [(1, 4), (7, 260), (8, 2048), (17, 1028)])
def test_f32_rows(ctx, tokens, rows, cols):
    """Row and token counts off the eight-row, eight-token tile; two parts with a cut inside one."""
    w = G.normal(90 + rows, rows + 2, cols)
    x = G.normal(91 + tokens, tokens, cols)
    a = ctx.matrix_upload(Q.GGML_F32, w.view(np.uint8), rows + 2, cols)
    got = ctx.matmul([(a, 0, rows), (a, rows, 2)], x, tokens, rows + 2)
    assert rel_l2(got, x.astype(np.float64) @ w.astype(np.float64).T) <= 1e-6
    ctx.matrix_free(a)
