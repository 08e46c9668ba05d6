"""GPU parity of the tcgen05 small-M GEMM (16 or more token rows per weight read) against the
CPU oracle's fused row dots. Weights and activations are rounded to fp16 on this path, so the
bound is the 1e-3 relative L2 of the GEMM outputs, with the measured error asserted tighter."""
import numpy as np
import pytest
import torch

from gufo_npu_b200 import quantize as Q
from gufo_npu_b200.backend import Context
from tests.golden import make_golden as G

pytestmark = pytest.mark.gpu

GEMM_TOL = 1e-3


def rel_l2(got, want):
    got = np.asarray(got, dtype=np.float64).ravel()
    want = np.asarray(want, dtype=np.float64).ravel()
    return float(np.linalg.norm(got - want) / max(np.linalg.norm(want), 1e-30))


@pytest.fixture(scope="module")
def ctx():
    """Every product of 16 or more token rows goes to the tcgen05 GEMM here (option value 2);
    by default the dispatcher keeps small batches on the 8-token passes where those are faster."""
    c = Context(0)
    c.set_option("tc_gemm", 2)
    yield c
    c.close()


def _weights(seed, rows, cols, ggml_type=Q.GGML_Q4_K):
    raw = Q.quantize(ggml_type, torch.from_numpy(G.normal(seed, rows, cols) * 0.02)).numpy()
    return raw.reshape(rows, -1)


@pytest.mark.parametrize("ggml_type", [Q.GGML_Q4_K, Q.GGML_Q6_K])
@pytest.mark.parametrize("rows,cols", [(256, 512), (130, 256), (1000, 2560), (2560, 9728)])
@pytest.mark.parametrize("tokens", [16, 17, 33, 128, 131])
def test_gemm_matches_oracle(ctx, oracle, ggml_type, rows, cols, tokens):
    """One Q4_K or Q6_K part: row counts off the 128-row tile, K shared by a cluster's thread blocks
    (1000 x 2560, 2560 x 9728), block counts that leave a partial slab in the Q6_K device arrangement (10, 38),
    token counts off the tile granule and past one pass."""
    if rows * cols * tokens > 1.5e9:
        tokens = min(tokens, 33)
    raw = _weights(40 + rows % 7, rows, cols, ggml_type)
    x = G.normal(50 + tokens, tokens, cols)
    m = ctx.matrix_upload(ggml_type, raw, rows, cols)
    got = ctx.matmul([(m, 0, rows)], x, tokens, rows)
    ctx.synchronize()
    want = oracle.matmul([(raw, ggml_type, 0, rows)], cols, x)
    err = rel_l2(got, want)
    assert err <= GEMM_TOL, err
    assert err <= 5e-4, err
    # Per token too: no row of the batch may hide behind the others.
    for t in range(tokens):
        assert rel_l2(got[t], want[t]) <= GEMM_TOL, t
    ctx.matrix_free(m)


def test_gemm_agrees_with_the_eight_token_passes(ctx):
    """The same product with the tensor-memory path switched off (int8 tensor-core passes of 8
    tokens) differs only by the fp16 rounding of this path."""
    rows, cols, tokens = 384, 1024, 40
    raw = _weights(61, rows, cols)
    x = G.normal(62, tokens, cols)
    m = ctx.matrix_upload(Q.GGML_Q4_K, raw, rows, cols)
    got = ctx.matmul([(m, 0, rows)], x, tokens, rows)
    ctx.set_option("tc_gemm", 0)
    try:
        ref = ctx.matmul([(m, 0, rows)], x, tokens, rows)
    finally:
        ctx.set_option("tc_gemm", 2)
    assert not np.array_equal(got, ref)
    assert rel_l2(got, ref) <= 5e-4
    ctx.matrix_free(m)


@pytest.mark.parametrize("ggml_type", [Q.GGML_Q4_K, Q.GGML_Q6_K])
@pytest.mark.parametrize("rows,blocks,tokens", [(128, 2, 17), (129, 3, 190), (200, 7, 200), (640, 13, 33), (2300, 8, 18)])
def test_gemm_units_shared_by_clusters(ctx, oracle, ggml_type, rows, blocks, tokens):
    """Units whose steps do not divide by the cluster, ragged last tiles, columns that do not divide
    by the cluster's owners, two token groups; outputs in the middle of wider rows. Twice alike, bit
    for bit: the shares are added in a fixed order."""
    cols = 256 * blocks
    raw = _weights(90 + blocks, rows, cols, ggml_type)
    x = torch.from_numpy(G.normal(91, tokens, cols)).cuda()
    m = ctx.matrix_upload(ggml_type, raw, rows, cols)
    y = torch.full((2, tokens, rows + 3), 7.0, device="cuda")
    torch.cuda.synchronize()
    for i in range(2):   # a second part of three rows: the rows of y are no multiple of 16 bytes
        ctx.matmul_device(Context._parts([(m, 0, rows), (m, 0, 3)]), 2, x, tokens, y[i])
    ctx.synchronize()
    assert torch.equal(y[0], y[1])
    want = oracle.matmul([(raw, ggml_type, 0, rows)], cols, x.cpu().numpy())
    assert rel_l2(y[0, :, :rows].cpu(), want) <= 5e-4
    assert torch.equal(y[0, :, rows:], y[0, :, :3])
    ctx.matrix_free(m)


def test_gemm_stacked_parts_and_row_ranges(ctx, oracle):
    """Gate and up stacked (one Q4_K, one Q6_K: two launches), a row range inside a matrix, an
    F32 part beside them (it takes the other kernels), every output column in its place."""
    cols, tokens = 768, 24
    gate, up = _weights(63, 300, cols), _weights(64, 300, cols, Q.GGML_Q6_K)
    extra = G.normal(65, 5, cols)
    mg = ctx.matrix_upload(Q.GGML_Q4_K, gate, 300, cols)
    mu = ctx.matrix_upload(Q.GGML_Q6_K, up, 300, cols)
    mf = ctx.matrix_upload(Q.GGML_F32, extra.view(np.uint8), 5, cols)
    x = G.normal(66, tokens, cols)
    got = ctx.matmul([(mg, 0, 300), (mf, 0, 5), (mu, 17, 200)], x, tokens, 505)
    want = oracle.matmul([(gate, Q.GGML_Q4_K, 0, 300), (extra.view(np.uint8).reshape(5, -1), Q.GGML_F32, 0, 5),
                          (up, Q.GGML_Q6_K, 17, 200)], cols, x)
    assert rel_l2(got[:, :300], want[:, :300]) <= 5e-4
    assert rel_l2(got[:, 300:305], want[:, 300:305]) <= 1e-5
    assert rel_l2(got[:, 305:], want[:, 305:]) <= 5e-4
    for m in (mg, mu, mf):
        ctx.matrix_free(m)


def test_gemm_ragged_verify_batch(ctx, oracle):
    """Config-5 packing at reduced width: 32 sequences of 1 to 4 draft tokens (seeded) packed into
    M rows with offsets[33]; each sequence's rows equal the same rows multiplied alone."""
    rng = np.random.default_rng(77)
    lengths = rng.integers(1, 5, size=32)
    offsets = np.concatenate([[0], np.cumsum(lengths)])
    m_rows = int(offsets[-1])
    rows, cols = 512, 1280
    raw = _weights(67, rows, cols)
    x = G.normal(68, m_rows, cols)
    m = ctx.matrix_upload(Q.GGML_Q4_K, raw, rows, cols)
    got = ctx.matmul([(m, 0, rows)], x, m_rows, rows)
    want = oracle.matmul([(raw, Q.GGML_Q4_K, 0, rows)], cols, x)
    for s in range(32):
        lo, hi = int(offsets[s]), int(offsets[s + 1])
        assert rel_l2(got[lo:hi], want[lo:hi]) <= GEMM_TOL, s
    ctx.matrix_free(m)


def test_gemm_activation_range(ctx, oracle):
    """Rows of very different magnitude in one batch: each row is scaled on its own, so a huge
    row does not flush a tiny one and neither overflows fp16. A zero row stays zero."""
    rows, cols, tokens = 256, 512, 16
    raw = _weights(69, rows, cols)
    x = G.normal(70, tokens, cols)
    x[1] *= 1e30
    x[2] *= 1e-30
    x[3] = 0.0
    x[4] *= 65504.0 * 4
    m = ctx.matrix_upload(Q.GGML_Q4_K, raw, rows, cols)
    got = ctx.matmul([(m, 0, rows)], x, tokens, rows)
    want = oracle.matmul([(raw, Q.GGML_Q4_K, 0, rows)], cols, x)
    assert np.isfinite(got).all()
    assert np.all(got[3] == 0.0)
    for t in range(tokens):
        if t != 3:
            assert rel_l2(got[t], want[t]) <= GEMM_TOL, t
    ctx.matrix_free(m)


def _near_float64(y, x, w):
    """y = x w^T to the rounding of weights and inputs to fp16: as a whole, and in every row and token.

    An output's size is taken as |w row| |x row| / sqrt(cols), what it is on average for inputs that
    are random: the outputs of a row at 17 tokens may by chance be small together (chi-squared of 17
    degrees, a sixth of its mean in the smallest of 19400 rows), its errors may not be large together
    (three times the mean in the largest: 1.7 x 4e-4)."""
    error = (y.double() - x.double() @ w.double().T) ** 2
    size = (x.double() ** 2).sum(1)[:, None] * (w.double() ** 2).sum(1)[None] / x.shape[1]
    assert float((error.sum() / size.sum()).sqrt()) <= 5e-4
    for d in (0, 1):
        assert float((error.sum(d) / size.sum(d)).sqrt().max()) <= GEMM_TOL, d


@pytest.mark.parametrize("ggml_type", [Q.GGML_Q4_K, Q.GGML_Q6_K])
@pytest.mark.parametrize("rows,cols,tokens", [
    (2560, 4096, 79), (2560, 9728, 128),        # clusters of six, 80 and 128 columns
    (2560, 9728, 352),                          # clusters of three, two groups of 176
    (2560, 4096, 512), (9000, 2560, 190),       # clusters of two, 176 and 192 columns; a ragged tile
    (12288, 2560, 128), (12288, 2560, 512),     # whole tiles, one round and two
    (19400, 2560, 17), (19400, 2560, 79),       # 152 tiles cut over 148 blocks, the last one ragged
    (19400, 2560, 352), (19456, 2560, 512),     # the same with two and three groups, ragged columns
    (12000, 9728, 17), (12000, 9728, 128),      # 94 tiles cut over 148 blocks: up to three shares a tile
])
def test_gemm_plans_against_float64(ctx, ggml_type, rows, cols, tokens):
    """Every way the planner cuts a product on 148 SMs, at narrow and wide token groups (few raw
    stages); twice, as the second run meets the counters and partial sums the first has left."""
    gen = torch.Generator("cuda").manual_seed(rows + tokens)
    raw = Q.quantize(ggml_type, torch.randn(rows, cols, device="cuda", generator=gen) * 0.02)
    x = torch.randn(tokens, cols, device="cuda", generator=gen)
    w = torch.empty(rows, cols, device="cuda")
    y = torch.full((2, tokens, rows), 7.0, device="cuda")
    torch.cuda.synchronize()
    m = ctx.matrix_from_device(ggml_type, raw.data_ptr(), rows, cols)
    ctx.dequantize_device(m, 0, rows, w)
    for i in range(2):
        ctx.matmul_device(Context._parts([(m, 0, rows)]), 1, x, tokens, y[i])
    ctx.synchronize()
    assert torch.equal(y[0], y[1])
    _near_float64(y[0], x, w)
    ctx.matrix_free(m)


def test_gemm_ring_of_two_blocks_under_load(ctx):
    """Wide token groups leave the raw blocks a ring of two stages, refilled from L2 by the groups
    behind the first: a stage must not be overwritten while lanes still read it. Many launches,
    all alike bit for bit (a row of weights from the next block differs in every token), and the
    first against float64."""
    rows, cols, tokens = 19456, 2560, 352   # two groups of 176
    raw = torch.randint(0, 256, (rows, cols // 256, 144), device="cuda", dtype=torch.uint8,
                        generator=torch.Generator("cuda").manual_seed(3))
    raw[:, :, 0:4] = torch.tensor([1e-3, 1e-3], device="cuda").half().view(torch.uint8)
    x = torch.randn(tokens, cols, device="cuda", generator=torch.Generator("cuda").manual_seed(4))
    y = torch.empty(12, tokens, rows, device="cuda")
    torch.cuda.synchronize()
    m = ctx.matrix_from_device(Q.GGML_Q4_K, raw.data_ptr(), rows, cols)
    for _ in range(8):
        for i in range(12):
            ctx.matmul_device(Context._parts([(m, 0, rows)]), 1, x, tokens, y[i])
        ctx.synchronize()
        for i in range(1, 12):
            assert torch.equal(y[0], y[i])
    w = torch.empty(rows, cols, device="cuda")
    torch.cuda.synchronize()
    ctx.dequantize_device(m, 0, rows, w)
    ctx.synchronize()
    _near_float64(y[0], x, w)
    ctx.matrix_free(m)


def _rows_whose_words_cancel(ggml_type, blocks, word, seed):
    """One row of `blocks` blocks whose bytes, as a dequantizing lane loads them for 64 of the values
    of a block (its head or its scales and d, and the words of the codes), have `word` as their xor."""
    rng = np.random.default_rng(seed)
    size = Q.BLOCK_BYTES[ggml_type]
    raw = rng.integers(0, 256, (blocks, size), dtype=np.uint8)
    d = np.float16(1e-3).tobytes()
    words = lambda a: np.ascontiguousarray(a).view(np.uint32)
    for block in raw:
        if ggml_type == Q.GGML_Q4_K:
            block[0:4] = np.frombuffer(d + d, np.uint8)
        else:
            block[208:210] = np.frombuffer(d, np.uint8)
        for p in range(4):
            if ggml_type == Q.GGML_Q4_K:
                codes = block[16 + 32 * p:48 + 32 * p]
                rest = words(block[0:16])
            else:
                h = p >> 1
                codes = block[64 * h + 32 * (p & 1):64 * h + 32 * (p & 1) + 32]
                rest = np.concatenate([words(block[128 + 32 * h:160 + 32 * h]), words(block[192 + 8 * h:200 + 8 * h]),
                                       np.array([int.from_bytes(d, "little")], np.uint32)])
            last = np.uint32(word) ^ np.bitwise_xor.reduce(rest) ^ np.bitwise_xor.reduce(words(codes[:28]))
            codes[28:32] = np.frombuffer(np.uint32(last).tobytes(), np.uint8)
            assert np.bitwise_xor.reduce(np.concatenate([rest, words(codes)])) == word
    return raw.reshape(-1)


@pytest.mark.parametrize("ggml_type", [Q.GGML_Q4_K, Q.GGML_Q6_K])
@pytest.mark.parametrize("word", [0x00000000, 0xFFFFFFFF, 0xDEADBEEF])
def test_gemm_raw_stages_are_released_whatever_the_bytes(ctx, ggml_type, word):
    """Equal rows, so that all lanes of a warp load the same words, with the xors a release could
    mistake for nothing loaded: 152 tiles of ten blocks, more steps a thread block than raw stages."""
    rows, blocks, tokens = 152 * 128, 10, 32
    cols = 256 * blocks
    one = _rows_whose_words_cancel(ggml_type, blocks, word, word & 0xFF)
    raw = torch.from_numpy(one).cuda().repeat(rows, 1)
    x = torch.randn(tokens, cols, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    w = torch.empty(1, cols, device="cuda")
    y = torch.full((tokens, rows), 7.0, device="cuda")
    torch.cuda.synchronize()
    m = ctx.matrix_from_device(ggml_type, raw.data_ptr(), rows, cols)
    ctx.dequantize_device(m, 0, 1, w)
    ctx.matmul_device(Context._parts([(m, 0, rows)]), 1, x, tokens, y)
    ctx.synchronize()
    want = (x.double() @ w.double().T).expand(tokens, rows)
    assert float((y.double() - want).norm() / want.norm()) <= GEMM_TOL
    ctx.matrix_free(m)
