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


@pytest.mark.parametrize("replaced", [False, True])
def test_scratch_of_a_context_that_changed_streams_is_not_handed_on(ctx, replaced):
    """Work may be left on the stream it was given first; of others the next context takes it over."""
    streams = [torch.cuda.Stream() for _ in range(2)]
    x, y = torch.randn(512, 2560, device="cuda:0"), torch.empty(512, 16, device="cuda:0")
    free = []
    for _ in range(2):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        own = Context(0, streams[0].cuda_stream)
        m, _ = _matrix(own, Q.GGML_Q4_K, 4096, 2560, 1)
        y = torch.empty(512, 4096, device="cuda:0")
        torch.cuda.synchronize()
        own.matmul_device([(m, 0, 4096)], None, x, 512, y)
        if replaced:
            own.set_stream(streams[1].cuda_stream)
        own.close()
        del y
        free.append((before - torch.cuda.mem_get_info()[0]) >> 20)
    assert free[1] <= 8 and (not replaced or free[0] <= 24), free


def test_f32_rows_of_more_tokens_than_a_grid_holds(ctx):
    dev = torch.device("cuda:0")
    tokens = 65535 * 8 + 3
    w = G.normal(5, 2, 4).astype(np.float32)
    m = ctx.matrix_upload(Q.GGML_F32, w.view(np.uint8), 2, 4)
    x, y = torch.randn(tokens, 4, device=dev), torch.empty(tokens, 2, device=dev)
    torch.cuda.synchronize()
    ctx.matmul_device([(m, 0, 2)], None, x, tokens, y)
    ctx.synchronize()
    want = x.double() @ torch.from_numpy(w).to(dev).double().T
    assert (y - want).abs().max() <= 1e-5
    ctx.matrix_free(m)


def test_gemm_scratch_is_bounded(ctx):
    """A product of a few rows takes little, one of many no more for ever more rows; those in passes
    are right."""
    own = Context(0)
    dev = torch.device("cuda:0")
    small, _ = _matrix(own, Q.GGML_Q4_K, 16, 256, 1)
    wide, w = _matrix(own, Q.GGML_Q4_K, 16, 9728, 2)
    x = torch.randn(12000, 9728, device=dev, generator=torch.Generator(device=dev).manual_seed(1))
    y = torch.empty(12000, 16, device=dev)

    def taken(m, tokens, cols):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        own.matmul_device([(m, 0, 16)], None, x, tokens, y)
        own.synchronize()
        return (before - torch.cuda.mem_get_info()[0]) >> 20
    assert taken(small, 17, 256) <= 4
    first = [taken(wide, tokens, 9728) for tokens in (3100, 6000)]
    assert sum(first) <= 200
    want = x[:6000].double() @ torch.from_numpy(w).to(dev).T
    assert rel_l2(y[:6000].cpu().numpy(), want.cpu().numpy()) <= 5e-4
    assert [taken(wide, tokens, 9728) for tokens in (1537, 4000, 9000, 12000)] == [0, 0, 0, 0]
    own.close()


@pytest.mark.parametrize("ggml_type", [Q.GGML_Q4_K, Q.GGML_Q6_K])
@pytest.mark.parametrize("tokens,rows,cols", [
    (2, 40, 2048), (3, 4752, 1280), (3, 33, 1536), (4, 4736, 2560), (5, 16, 2048), (8, 17, 256), (8, 4753, 1280), (6, 31, 1792),
])
def test_few_rows_converted_in_the_product_or_ahead_of_it(ctx, ggml_type, tokens, rows, cols):
    """Either side of the line between the two (16 and 40 blocks of 256 values, 4736 rows)."""
    m, w = _matrix(ctx, ggml_type, rows, cols, 60 + rows % 7)
    x = G.normal(61 + tokens, tokens, cols)
    got = ctx.matmul([(m, 0, rows)], x, tokens, rows)
    want = x.astype(np.float64) @ w.T
    assert rel_l2(got, want) <= 2e-6
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


@pytest.mark.parametrize("nseq,key_heads,value_heads,head_dim", [(1, 16, 16, 128), (2, 2, 4, 32), (3, 2, 4, 64), (16, 2, 2, 96),
                                                                (17, 8, 8, 128), (64, 4, 8, 128), (65, 1, 3, 64)])
@pytest.mark.parametrize("out_of_place", [False, True])
def test_delta_rule_over_launch_sizes(ctx, nseq, key_heads, value_heads, head_dim, out_of_place):
    """Sequences on either side of what a launch's arguments hold, head dims off the models', rows off
    a 16-byte boundary, in float64."""
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(nseq)

    def rand(*shape):   # one float past an aligned address
        n = int(np.prod(shape))
        return torch.randn(n + 1, device=dev, generator=gen)[1:].reshape(shape)
    unit = torch.nn.functional.normalize
    state = torch.randn(nseq, value_heads, head_dim, head_dim, device=dev, generator=gen) * 0.1
    before, out = state.double(), torch.zeros_like(state)
    q, k, v = rand(nseq, key_heads, head_dim), rand(nseq, key_heads, head_dim), rand(nseq, value_heads, head_dim)
    q.copy_(unit(q.clone(), dim=-1)), k.copy_(unit(k.clone(), dim=-1))
    decay, beta, y = rand(nseq, value_heads).sigmoid(), rand(nseq, value_heads).sigmoid(), rand(nseq, value_heads, head_dim)
    seqs = [dict(state=state[i], state_out=out[i] if out_of_place else None, q=q[i], k=k[i], v=v[i], decay=decay[i],
                 beta=beta[i], y=y[i]) for i in range(nseq)]
    torch.cuda.synchronize()
    ctx.delta_rule_device(seqs, key_heads, value_heads, head_dim)
    ctx.synchronize()
    of = torch.arange(value_heads, device=dev) % key_heads
    kk, qq = k.double()[:, of], q.double()[:, of]
    want = before * decay.double()[..., None, None]
    delta = beta.double()[..., None] * (v.double() - torch.einsum("nhij,nhi->nhj", want, kk))
    want = want + kk[..., None] * delta[..., None, :]
    assert rel_l2((out if out_of_place else state).cpu().numpy(), want.cpu().numpy()) <= 2e-7
    assert rel_l2(y.cpu().numpy(), torch.einsum("nhij,nhi->nhj", want, qq).cpu().numpy()) <= 4e-7
    if out_of_place:
        assert torch.equal(state.double(), before)


@pytest.mark.parametrize("head_dim,conv_kernel,nseq", [(32, 2, 3), (64, 8, 5), (128, 4, 66), (128, 5, 3)])
def test_mixer_run_of_many_sequences_equals_one_token_at_a_time(ctx, oracle, head_dim, conv_kernel, nseq):
    """Sequences of one to four tokens together (more than one launch's worth in one case), bit for
    bit against one sequence and token at a time; one of those against the oracle."""
    from gufo_npu_b200 import synth
    from gufo_npu_b200.backend import CudaMixer
    from tests.test_oracle import _deltanet_cfg, _deltanet_weights
    dev = torch.device("cuda:0")
    cfg = synth.ModelConfig(layers=1, hidden=512, ffn=256, vocab=256, linear_key_heads=2, linear_value_heads=4,
                            linear_head_dim=head_dim, conv_kernel=conv_kernel)
    if cfg.value_dim % 256:
        cfg.proj_type = Q.GGML_F32
    tensors = synth.build_model(cfg, 5)
    mixer = CudaMixer(ctx, cfg, tensors)
    gen = torch.Generator(device=dev).manual_seed(11)
    counts = [1 + i % 4 for i in range(nseq)]
    width = cfg.conv_channels + cfg.value_dim + 2 * cfg.linear_value_heads

    def rand(*shape):
        return torch.randn(*shape, device=dev, generator=gen)
    seqs = [{"n_tokens": n, "in": rand(n, width), "h": rand(n, cfg.hidden), "conv_in": rand(mixer.conv_values()),
             "conv_out": rand(mixer.conv_values()), "conv_saved": rand(mixer.conv_values()),
             "ssm": rand(mixer.ssm_values()) * 0.1, "ssm_spec": rand(mixer.ssm_values()),
             "y": rand(n, cfg.value_dim)} for n in counts]
    before = [(q["conv_in"].clone(), q["ssm"].clone()) for q in seqs]
    torch.cuda.synchronize()
    mixer.Run(0, seqs)
    ctx.synchronize()
    for i in sorted({0, 1, 2, nseq // 2, nseq - 1}):
        q, n = seqs[i], counts[i]
        conv, ssm = before[i]
        for t in range(n):
            one = {"n_tokens": 1, "in": q["in"][t:t + 1], "h": q["h"][t:t + 1], "conv_in": conv,
                   "conv_out": torch.empty_like(conv), "ssm": ssm.clone(), "y": torch.empty(1, cfg.value_dim, device=dev)}
            torch.cuda.synchronize()
            mixer.Run(0, [one])
            ctx.synchronize()
            assert torch.equal(one["y"][0], q["y"][t]), (i, t)
            if t == n - 1:
                assert torch.equal(one["ssm"], q["ssm_spec"] if n > 1 else q["ssm"])
                assert torch.equal(one["conv_out"], q["conv_out"])
                assert n == 1 or (torch.equal(ssm, q["ssm"]) and torch.equal(conv, q["conv_saved"]))
            conv, ssm = one["conv_out"], one["ssm"]
    # Mixer::Linear (gates in the input row) of the same shape against the oracle.
    x, conv, ssm = rand(3, width), rand(3, mixer.conv_values()), rand(3, mixer.ssm_values()) * 0.1
    host = [(x[s].cpu().numpy(), conv[s].cpu().numpy().copy(), ssm[s].cpu().numpy().copy()) for s in range(3)]
    out, y = torch.empty_like(conv), torch.empty(3, cfg.value_dim, device=dev)
    torch.cuda.synchronize()
    mixer.Linear(0, [{"in": x[s], "conv_in": conv[s], "conv_out": out[s], "ssm": ssm[s], "y": y[s]} for s in range(3)])
    ctx.synchronize()
    for s, (hx, hconv, hssm) in enumerate(host):
        want, _ = oracle.deltanet_linear(_deltanet_cfg(cfg), _deltanet_weights(cfg, tensors, 0), hx, hconv, hssm)
        assert rel_l2(y[s].cpu().numpy(), want) <= 1e-4
        assert rel_l2(ssm[s].cpu().numpy(), hssm) <= 1e-4


@pytest.mark.parametrize("inplace", [False, True])
def test_mixer_run_inside_a_first_capture_and_over_its_own_input(inplace):
    """Three sequences captured by a context that has run nothing, and outputs laid over z: the bits of
    a plain call."""
    from gufo_npu_b200 import synth
    from gufo_npu_b200.backend import CudaMixer
    dev = torch.device("cuda:0")
    cfg = synth.ModelConfig(layers=1, hidden=512, ffn=256, vocab=256, linear_key_heads=2, linear_value_heads=4)
    tensors = synth.build_model(cfg, 5)
    width, z_at = cfg.conv_channels + cfg.value_dim + 2 * cfg.linear_value_heads, cfg.conv_channels
    gen = torch.Generator(device=dev).manual_seed(2)

    def rand(*shape):
        return torch.randn(*shape, device=dev, generator=gen)
    results = []
    first = [(rand(2, width), rand(2, cfg.hidden)) for _ in range(3)]
    for captured in (False, True):
        stream = torch.cuda.Stream()
        own = Context(0, stream.cuda_stream)
        mixer = CudaMixer(own, cfg, tensors)
        gen.manual_seed(7)
        seqs = []
        for row, h in first:
            row = row.clone()
            seqs.append({"n_tokens": 2, "in": row, "h": h, "conv_in": rand(mixer.conv_values()),
                         "conv_out": rand(mixer.conv_values()), "conv_saved": rand(mixer.conv_values()),
                         "ssm": rand(mixer.ssm_values()) * 0.1, "ssm_spec": rand(mixer.ssm_values()),
                         "y": row[:, z_at:z_at + cfg.value_dim] if inplace and captured else
                         torch.empty(2, cfg.value_dim, device=dev)})
        torch.cuda.synchronize()
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                mixer.Run(0, seqs)
            graph.replay()
        else:
            mixer.Run(0, seqs)
        torch.cuda.synchronize()
        results.append([torch.cat([q[key].reshape(-1) for q in seqs]) for key in ("y", "ssm", "ssm_spec", "conv_out")])
        del mixer
        own.close()
    for a, b in zip(*results):
        assert torch.equal(a, b)


def _random_rows(ctx, ggml_type, rows, cols, seed):
    """Any code bytes beside small fp16 scales: a matrix handle and its values in float64."""
    rng = np.random.default_rng(seed)
    per, size = Q.BLOCK_ELEMENTS[ggml_type], Q.BLOCK_BYTES[ggml_type]
    raw = rng.integers(0, 256, (rows * cols // per, size), dtype=np.uint8)
    for at in ((0, 2) if ggml_type == Q.GGML_Q5_K else (0,)):
        raw[:, at:at + 2] = (1e-3 * (1.0 + rng.random(raw.shape[0]))).astype(np.float16).view(np.uint8).reshape(-1, 2)
    m = ctx.matrix_upload(ggml_type, raw.reshape(rows, -1), rows, cols)
    return m, ctx.dequantize(m, 0, rows, cols).astype(np.float64)


@pytest.mark.parametrize("ggml_type", [Q.GGML_Q5_K, Q.GGML_Q8_0])
@pytest.mark.parametrize("tokens", [1, 2, 3, 5, 8, 9])
@pytest.mark.parametrize("rows,cols", [(1, 256), (7, 2048), (133, 2304), (6, 9728)])
def test_q5_and_q8_rows_split_over_warps(ctx, ggml_type, tokens, rows, cols):
    """Row and token counts off the tile, K shorter and longer than a round of the warps; two parts
    with a cut inside one."""
    m, w = _random_rows(ctx, ggml_type, rows + 2, cols, 50 + rows)
    x = G.normal(51 + tokens, tokens, cols)
    got = ctx.matmul([(m, 0, rows), (m, rows, 2)], x, tokens, rows + 2)
    want = x.astype(np.float64) @ w.T
    assert rel_l2(got, want) <= 1e-6
    ctx.matrix_free(m)


@pytest.mark.parametrize("tokens,rows,cols", [(1, 16384, 256), (1, 16385, 256), (8, 9000, 512), (40, 7000, 8192), (3, 5, 768)])
def test_host_rows_pinned_and_pageable(ctx, tokens, rows, cols):
    """Host inputs and results on either side of the sizes that are staged, stored directly or left to
    the driver's copy, in pageable and in pinned memory: the same bytes."""
    m, w = _matrix(ctx, Q.GGML_Q4_K, rows, cols, 41)
    x = G.normal(42, tokens, cols).astype(np.float32)
    got = ctx.matmul([(m, 0, rows)], x, tokens, rows)
    assert rel_l2(got, x.astype(np.float64) @ w.T) <= 1e-3
    kept = got.copy()
    parts = Context._parts([(m, 0, rows)])
    px, py = torch.from_numpy(x).pin_memory(), torch.empty(tokens, rows).pin_memory()
    y = np.empty((tokens, rows), dtype=np.float32)
    for xa, ya, out in ((px.data_ptr(), y.ctypes.data, y), (px.data_ptr(), py.data_ptr(), py.numpy()),
                        (x.ctypes.data, py.data_ptr(), py.numpy())):
        out[:] = 0
        ctx.matmul_host(parts, 1, xa, tokens, ya)
        assert np.array_equal(out, kept)
    other = ctx.matmul([(m, 0, rows)], 2 * x, tokens, rows)
    assert np.array_equal(got, kept) and not np.shares_memory(got, other)
    ctx.matrix_free(m)


@pytest.mark.parametrize("tokens,rows,cols", [(1, 9000, 256), (8, 9000, 512), (3, 700, 12288)])
def test_host_rows_that_are_pinned_in_part_or_off_a_float(ctx, tokens, rows, cols):
    """Buffers of which the first pages are registered, and ones that start inside a float: copied, the
    same bytes. The step's logits likewise, but for the first, which the driver does not copy to."""
    import mmap
    from gufo_npu_b200 import _capi, synth
    from gufo_npu_b200.backend import CudaDecoder, CudaProjections
    rt = torch.cuda.cudart()
    m, w = _matrix(ctx, Q.GGML_Q4_K, rows, cols, 41)
    x = G.normal(42, tokens, cols).astype(np.float32)
    parts = Context._parts([(m, 0, rows)])
    want = ctx.matmul([(m, 0, rows)], x, tokens, rows)
    assert rel_l2(want, x.astype(np.float64) @ w.T) <= 1e-3
    for registered, shift in ((4096, 0), (1 << 20, 2), (1 << 20, 4), (0, 1)):
        buffers = [mmap.mmap(-1, 2 << 20) for _ in range(2)]
        bx, by = (np.frombuffer(b, dtype=np.uint8) for b in buffers)
        if registered:
            assert int(rt.cudaHostRegister(bx.ctypes.data, registered, 0)) == 0
            assert int(rt.cudaHostRegister(by.ctypes.data, registered, 0)) == 0
        bx[shift:shift + x.nbytes] = x.view(np.uint8).ravel()
        ctx.matmul_host(parts, 1, bx.ctypes.data + shift, tokens, by.ctypes.data + shift)
        got = by[shift:shift + want.nbytes].tobytes()
        if registered:
            assert int(rt.cudaHostUnregister(bx.ctypes.data)) == 0 and int(rt.cudaHostUnregister(by.ctypes.data)) == 0
        assert got == want.tobytes()
    ctx.matrix_free(m)
    if tokens == 1:
        cfg = synth.ModelConfig(layers=4, hidden=256, ffn=512, vocab=40000, heads=2, kv_heads=1, head_dim=128, rope_dim=32,
                                linear_key_heads=2, linear_value_heads=4, linear_head_dim=128)
        tensors = synth.build_model(cfg, 3)
        dec = CudaDecoder(CudaProjections(ctx, cfg, tensors), tensors, max_positions=64)
        want = dec.Step(7)
        for registered, shift in ((4096, 0), (1 << 20, 2)):   # the first: no copy reaches it either
            dec.Reset()
            buffer = mmap.mmap(-1, 2 << 20)
            b = np.frombuffer(buffer, dtype=np.uint8)
            assert int(rt.cudaHostRegister(b.ctypes.data, registered, 0)) == 0
            if shift == 0:
                with pytest.raises(_capi.GufoCudaError):
                    dec.Step(7, b.ctypes.data)
            else:
                dec.Step(7, b.ctypes.data + shift)
                assert b[shift:shift + want.nbytes].tobytes() == want.tobytes()
            ctx.synchronize()
            assert int(rt.cudaHostUnregister(b.ctypes.data)) == 0
        dec.close()


@pytest.mark.parametrize("context_first", [False, True])
def test_decoder_and_context_closed_in_either_order(context_first):
    """All memory comes back, and a decoder whose context has gone refuses to step."""
    from gufo_npu_b200 import _capi, synth
    from gufo_npu_b200.backend import CudaDecoder, CudaProjections
    cfg = synth.ModelConfig(layers=4, hidden=256, ffn=512, vocab=512, heads=2, kv_heads=1, head_dim=128, rope_dim=32,
                            linear_key_heads=2, linear_value_heads=4, linear_head_dim=128)
    tensors = synth.build_model(cfg, 3)
    free = []
    for _ in range(4):
        own = Context(0)
        dec = CudaDecoder(CudaProjections(own, cfg, tensors), tensors, max_positions=1 << 17)   # 64 MB of cache
        for token in (5, 6, 7, 8):
            dec.Step(token)
        if context_first:
            own.close()
            for call in (lambda: dec.Step(9), lambda: dec.StepTokens([9, 10]), dec.Reset, lambda: dec.Resolve(True),
                         lambda: dec.step_device(9)):
                with pytest.raises(_capi.GufoCudaError, match="context"):
                    call()
        dec.close()
        dec.close()
        own.close()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[-1] < 16 << 20, free


@pytest.mark.parametrize("vocab", [512, 40000])
def test_step_logits_in_any_memory(ctx, vocab):
    """Logits left on the device (many steps, none waited for), in pageable, pooled
    and alternating pinned memory: the same bits; pairs to the rounding of another order of sums."""
    from gufo_npu_b200 import synth
    from gufo_npu_b200.backend import CudaDecoder, CudaProjections
    cfg = synth.ModelConfig(layers=4, hidden=256, ffn=512, vocab=vocab, heads=2, kv_heads=1, head_dim=128, rope_dim=32,
                            linear_key_heads=2, linear_value_heads=4, linear_head_dim=128)
    tensors = synth.build_model(cfg, 3)
    dec = CudaDecoder(CudaProjections(ctx, cfg, tensors), tensors, max_positions=64, use_graph=True)
    tokens = [(37 * i + 11) % vocab for i in range(24)]
    want = []
    for t in tokens:
        at = dec.step_device(t)
        want.append(ctx.download(at, vocab))
    dec.Reset()
    for t in tokens:
        at = dec.step_device(t)
    assert np.array_equal(ctx.download(at, vocab), want[-1])
    dec.Reset()
    pinned = [torch.empty(vocab).pin_memory() for _ in range(2)]
    held = []
    for i, t in enumerate(tokens):
        if i % 4 == 3:
            got = dec.Step(t)
        elif i % 4 == 2:
            got = dec.Step(t, np.empty(vocab, dtype=np.float32))
        else:
            got = dec.Step(t, pinned[i % 2]).numpy().copy()
        held.append(got)
    for got, w in zip(held, want):
        assert np.array_equal(got, w)
    dec.Reset()
    for i in range(0, 16, 2):
        got = dec.StepTokens(tokens[i:i + 2])
        assert rel_l2(got[0], want[i]) <= 5e-4 and rel_l2(got[1], want[i + 1]) <= 5e-4
        dec.Resolve(True)
    dec.Reset()
    for i in range(8):
        got = dec.StepTokens([tokens[i], tokens[(i + 5) % 8]])
        assert rel_l2(got[0], want[i]) <= 5e-4
        dec.Resolve(False)
    dec.close()


@pytest.mark.parametrize("experts,k", [(8, 8), (33, 4), (256, 8), (257, 3), (1024, 40)])
def test_route_ties_and_counts(ctx, oracle, experts, k):
    """Expert counts off the warp and block widths, equal logits among the best, more slots than lanes."""
    dev = torch.device("cuda:0")
    tokens = 3
    logits = G.normal(31 + experts, tokens, experts + 1).astype(np.float32)
    logits[1, : experts // 2] = 2.5          # ties: the lower id first
    logits[2, experts // 3] = 1e4            # every other probability underflows
    x = torch.from_numpy(logits).to(dev)
    chosen = torch.empty(tokens, k, dtype=torch.int32, device=dev)
    weights = torch.empty(tokens, k, device=dev)
    scale = torch.empty(tokens, device=dev)
    torch.cuda.synchronize()
    ctx.route_device(x, experts + 1, tokens, experts, k, chosen, weights, scale)
    ctx.synchronize()
    for t in range(tokens):
        p = np.exp(logits[t, :experts].astype(np.float64) - float(logits[t, :experts].max()))
        order = np.lexsort((np.arange(experts), -p))[:k]
        assert chosen[t].cpu().numpy().tolist() == order.tolist()
        picked = p[order] / p.sum()
        assert rel_l2(weights[t].cpu().numpy(), picked / max(picked.sum(), 6.103515625e-5)) <= 1e-6


@pytest.mark.parametrize("experts,k", [(7, 7), (64, 8), (300, 8)])
def test_route_of_logits_that_are_not_finite(ctx, experts, k):
    """The ids stay distinct and below `experts` (the products address by them); the weights are NaN."""
    dev = torch.device("cuda:0")
    nan, inf = float("nan"), float("inf")
    logits = torch.randn(6, experts + 1, device=dev, generator=torch.Generator(device=dev).manual_seed(experts))
    logits[0, :experts] = nan
    logits[1, 3] = nan
    logits[2, 5] = inf
    logits[3, :experts - 2] = nan
    logits[4, :experts] = -inf
    chosen = torch.full((6, k), -7, dtype=torch.int32, device=dev)
    weights, scale = torch.zeros(6, k, device=dev), torch.zeros(6, device=dev)
    torch.cuda.synchronize()
    ctx.route_device(logits, experts + 1, 6, experts, k, chosen, weights, scale)
    ctx.synchronize()
    for row in chosen.cpu().tolist():
        assert min(row) >= 0 and max(row) < experts and len(set(row)) == k
    assert weights[:5].isnan().all() and torch.isfinite(weights[5]).all() and torch.isfinite(scale).all()


@pytest.mark.parametrize("heads,kv_heads,head_dim,rope_dim", [(8, 1, 64, 64), (3, 3, 128, 32), (16, 4, 256, 64),
                                                              (2, 1, 256, 0), (5, 1, 128, 128)])
@pytest.mark.parametrize("positions", [1, 2, 17, 64, 65, 128, 129, 193, 1000, 4099, 9001])
def test_attention_chunks_and_splits(ctx, heads, kv_heads, head_dim, rope_dim, positions):
    """Lengths around a chunk, around what one block takes and with a ragged last slice, in float64;
    a later call finds the arrival counters as it needs them."""
    import ctypes as C
    from gufo_npu_b200 import _capi
    dev = torch.device("cuda:0")
    hd, group, pos = head_dim, heads // kv_heads, positions - 1
    gen = torch.Generator(device=dev).manual_seed(positions)

    def rand(*shape):
        return torch.randn(*shape, device=dev, generator=gen)
    keys, values = rand(positions + 3, kv_heads * hd).half(), rand(positions + 3, kv_heads * hd).half()
    row, wq, wk = rand(2 * heads * hd + 2 * kv_heads * hd), 1 + 0.1 * rand(hd), 1 + 0.1 * rand(hd)
    row[:2 * hd] *= 1e-3   # a head far smaller than the others
    freq = (1.0 / 1e4 ** (2.0 * torch.arange(max(rope_dim // 2, 1), device=dev, dtype=torch.float64) / max(rope_dim, 1))).float()
    position = torch.tensor([pos], dtype=torch.int32, device=dev)
    queries, partials = torch.empty(heads * hd, device=dev), torch.empty(kv_heads * 32 * group * (hd + 2), device=dev)
    out = torch.empty(heads * hd, device=dev)
    args = _capi.AttentionArgs(heads, kv_heads, hd, rope_dim, positions + 3, 1e-6,
                               *[t.data_ptr() for t in (position, row, wq, wk, freq, keys, values, queries, partials, out)])
    torch.cuda.synchronize()
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        ctx._check(ctx.lib.gufo_cuda_attention_device(ctx.handle, C.byref(args)))
        ctx.synchronize()

    def head(x, w):
        x = x.double()
        x = x / torch.sqrt((x * x).mean() + 1e-6) * w.double()
        half = rope_dim // 2
        if half:
            angle = pos * freq[:half].double()
            lo, hi = x[:half].clone(), x[half:2 * half].clone()
            x[:half] = lo * torch.cos(angle) - hi * torch.sin(angle)
            x[half:2 * half] = lo * torch.sin(angle) + hi * torch.cos(angle)
        return x
    q_gate = row[:2 * heads * hd].reshape(heads, 2, hd)
    k_new = row[2 * heads * hd:][:kv_heads * hd].reshape(kv_heads, hd)
    v_new = row[2 * heads * hd + kv_heads * hd:].reshape(kv_heads, hd)
    K, V = keys.double().reshape(-1, kv_heads, hd), values.double().reshape(-1, kv_heads, hd)
    want = torch.empty(heads, hd, dtype=torch.float64, device=dev)
    for h in range(heads):
        kh = h // group
        assert (K[pos, kh] - head(k_new[kh], wk)).abs().max() <= 2e-3 * K[pos, kh].abs().max()
        assert torch.equal(V[pos, kh], v_new[kh].half().double())
        p = torch.softmax(K[:positions, kh] @ head(q_gate[h, 0], wq) / hd ** 0.5, 0)
        want[h] = (p @ V[:positions, kh]) * torch.sigmoid(q_gate[h, 1].double())
    assert rel_l2(out.cpu().numpy(), want.cpu().numpy()) <= 2e-6
    for h in range(heads):
        assert rel_l2(out.reshape(heads, hd)[h].cpu().numpy(), want[h].cpu().numpy()) <= 5e-6, h


def _attention_call(positions, heads, kv_heads, hd, seed):
    """Tensors of one attention call on random rows, the last of them its output, and its arguments."""
    from gufo_npu_b200 import _capi
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(seed)

    def rand(*shape):
        return torch.randn(*shape, device=dev, generator=gen)
    tensors = [torch.tensor([positions - 1], dtype=torch.int32, device=dev), rand(2 * (heads + kv_heads) * hd),
               1 + 0.1 * rand(hd), 1 + 0.1 * rand(hd), 0.1 + rand(16).abs(), rand(positions, kv_heads * hd).half(),
               rand(positions, kv_heads * hd).half(), torch.empty(heads * hd, device=dev),
               torch.empty(32 * heads * (hd + 2), device=dev), torch.empty(heads * hd, device=dev)]
    return tensors, _capi.AttentionArgs(heads, kv_heads, hd, 32, positions, 1e-6, *[t.data_ptr() for t in tensors])


def test_attention_in_used_scratch_with_more_kv_heads_than_before(ctx):
    """A context that takes over another's scratch, its first call on one KV head, the next on four."""
    import ctypes as C
    other = Context(0)
    m, _ = _matrix(other, Q.GGML_Q4_K, 4752, 1280, 3)
    other.matmul([(m, 0, 4752)], G.normal(4, 8, 1280), 8, 4752)   # leaves bytes in a block of 256 KB
    other.close()
    own = Context(0)
    outs = []
    for heads, kv_heads, hd in ((2, 1, 128), (4, 4, 64)):
        for use in (own, ctx):
            tensors, args = _attention_call(300, heads, kv_heads, hd, 1)
            torch.cuda.synchronize()
            for general in (0, 1):
                use.set_option("general_gemv", general)
                use._check(use.lib.gufo_cuda_attention_device(use.handle, C.byref(args)))
                use.synchronize()
                outs.append(tensors[-1].clone())
            use.set_option("general_gemv", 0)
            assert rel_l2(outs[-2].cpu().numpy(), outs[-1].cpu().numpy()) <= 2e-6
    own.close()


def _attention_in_float64(tensors, args):
    """The outputs from the fp16 rows as they are in the cache after the call."""
    position, row, wq, _, freq, keys, values = tensors[:7]
    heads, kv_heads, hd, half, pos = args.heads, args.kv_heads, args.head_dim, args.rope_dim // 2, int(position)
    q_gate = row[:2 * heads * hd].double().reshape(heads, 2, hd)
    q = q_gate[:, 0] / torch.sqrt((q_gate[:, 0] ** 2).mean(1, keepdim=True) + args.rms_eps) * wq.double()
    angle = pos * freq[:half].double()
    lo, hi = q[:, :half].clone(), q[:, half:2 * half].clone()
    q[:, :half] = lo * torch.cos(angle) - hi * torch.sin(angle)
    q[:, half:2 * half] = lo * torch.sin(angle) + hi * torch.cos(angle)
    of = torch.arange(heads, device=row.device) // (heads // kv_heads)
    k = keys[:pos + 1].double().reshape(-1, kv_heads, hd)[:, of]
    v = values[:pos + 1].double().reshape(-1, kv_heads, hd)[:, of]
    p = torch.softmax(torch.einsum("nhd,hd->hn", k, q) / hd ** 0.5, 1)
    return torch.einsum("hn,nhd->hd", p, v) * torch.sigmoid(q_gate[:, 1])


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(8, 2, 256), (2, 1, 128), (4, 4, 64)])
@pytest.mark.parametrize("positions", [100, 4096, 16384])
def test_attention_is_as_close_to_float64_as_fp32_arithmetic(ctx, heads, kv_heads, head_dim, positions):
    """The mean of six inputs. With fp32 arithmetic in place of the tensor core 1.8e-7 to 2.9e-7 was
    measured over these shapes; sums accumulated inside it: up to 6.5e-7."""
    import ctypes as C
    errors = []
    for seed in range(6):
        tensors, args = _attention_call(positions, heads, kv_heads, head_dim, seed)
        torch.cuda.synchronize()
        ctx._check(ctx.lib.gufo_cuda_attention_device(ctx.handle, C.byref(args)))
        ctx.synchronize()
        errors.append(rel_l2(tensors[-1].cpu().numpy(), _attention_in_float64(tensors, args).cpu().numpy()))
    assert np.mean(errors) <= 3.5e-7, errors


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(8, 2, 256), (2, 1, 128), (4, 4, 64)])
@pytest.mark.parametrize("positions", [1, 60, 700])
@pytest.mark.parametrize("what", ["value", "own value", "key", "keys", "own key", "query"])
def test_attention_over_cache_rows_that_are_not_finite(ctx, heads, kv_heads, head_dim, positions, what):
    """An infinite cache element (an fp16 overflow) reaches what it reaches in exact arithmetic, and no
    more."""
    import ctypes as C
    tensors, args = _attention_call(positions, heads, kv_heads, head_dim, 3)
    row, keys, values = tensors[1], tensors[5], tensors[6]
    at = positions // 2
    if what == "value":
        values[at, 5] = float("inf")
    elif what == "own value":
        row[2 * heads * head_dim + kv_heads * head_dim + 7] = -1e9
    elif what == "key":
        keys[at, 40] = float("inf")
    elif what == "keys":     # the first half of the slices
        keys[:at + 1, 40] = -float("inf")
    elif what == "own key":
        tensors[3][40] = 1e9
    else:
        row[3] = float("inf")
    torch.cuda.synchronize()
    ctx._check(ctx.lib.gufo_cuda_attention_device(ctx.handle, C.byref(args)))
    ctx.synchronize()
    got, want = tensors[-1].double(), _attention_in_float64(tensors, args).reshape(-1)
    assert torch.equal(want.isnan(), got.isnan())
    assert torch.equal(want[want.isinf()], got[want.isinf()])
    finite = torch.isfinite(want)
    assert torch.isfinite(got[finite]).all() and rel_l2(got[finite].cpu().numpy(), want[finite].cpu().numpy()) <= 2e-6


def test_attention_on_two_streams_and_in_concurrent_graphs():
    """Calls of one context that may be in flight together, on two streams and in two graphs captured
    by a context that has run none: each has the bits of a call by itself."""
    import ctypes as C
    shapes = [(9001, 8, 2, 256), (3000, 8, 2, 256), (700, 2, 1, 128), (16000, 16, 4, 64)]
    calls = [_attention_call(*shapes[i % 4], i) for i in range(16)]
    streams = [torch.cuda.Stream() for _ in range(2)]

    def run(own, args):
        own._check(own.lib.gufo_cuda_attention_device(own.handle, C.byref(args)))
    own = Context(0)
    want = []
    for tensors, args in calls:
        torch.cuda.synchronize()
        run(own, args)
        own.synchronize()
        want.append(tensors[-1].clone())
        tensors[-1].zero_()
    torch.cuda.synchronize()
    for _ in range(4):
        for i, (_, args) in enumerate(calls):
            own.set_stream(streams[i % 2].cuda_stream)
            run(own, args)
    torch.cuda.synchronize()
    for (tensors, _), w in zip(calls, want):
        assert torch.equal(tensors[-1], w)
        tensors[-1].zero_()
    own.close()
    own = Context(0, streams[0].cuda_stream)
    graphs = []
    for half in range(2):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=streams[0]):
            for _, args in calls[half::2]:
                run(own, args)
    for _ in range(4):
        for graph, stream in zip(graphs, streams):
            with torch.cuda.stream(stream):
                graph.replay()
    torch.cuda.synchronize()
    for (tensors, _), w in zip(calls, want):
        assert rel_l2(tensors[-1].cpu().numpy(), w.cpu().numpy()) <= 2e-6   # other slices in a graph
    own.close()


@pytest.mark.parametrize("ggml_type", [Q.GGML_Q4_K, Q.GGML_Q6_K])
@pytest.mark.parametrize("tokens,rows,cols", [
    (1, 20000, 2560), (2, 33, 256), (2, 20011, 768), (3, 16, 9728), (5, 9001, 2304), (8, 40, 2816), (8, 1500, 9728),
    (4, 12000, 512), (7, 2560, 4096),
])
def test_units_of_ragged_rows(ctx, ggml_type, tokens, rows, cols):
    """Fewer blocks a row than warps, rounds that end inside a tile, rows off the tile, several tiles
    a thread block, clusters, and more tokens than fit one pass."""
    m, w = _matrix(ctx, ggml_type, rows, cols, 20 + cols % 13)
    x = G.normal(21 + tokens, tokens, cols)
    got = ctx.matmul([(m, 0, rows)], x, tokens, rows)
    want = x.astype(np.float64) @ w.T
    assert rel_l2(got, want) <= 2e-6
    for t in range(tokens):
        assert rel_l2(got[t], want[t]) <= 4e-6, t
    ctx.matrix_free(m)


@pytest.mark.parametrize("ggml_type,tokens,cols", [(Q.GGML_Q4_K, 8, 5376), (Q.GGML_Q4_K, 7, 6144), (Q.GGML_Q4_K, 5, 8960),
                                                  (Q.GGML_Q6_K, 8, 5120), (Q.GGML_Q6_K, 7, 5888), (Q.GGML_Q6_K, 5, 8192)])
def test_widest_rows_of_one_pass(ctx, ggml_type, tokens, cols):
    """The rows go over the weights once: a launch that converts them and one that multiplies."""
    m, w = _matrix(ctx, ggml_type, 4800, cols, 9)
    x = torch.from_numpy(G.normal(10, tokens, cols).astype(np.float32)).to("cuda:0")
    y = torch.empty(tokens, 4800, device="cuda:0")
    torch.cuda.synchronize()
    before = ctx.launch_count()
    ctx.matmul_device([(m, 0, 4800)], None, x, tokens, y)
    assert ctx.launch_count() - before == 2
    ctx.synchronize()
    assert rel_l2(y.cpu().numpy(), x.cpu().numpy().astype(np.float64) @ w.T) <= 2e-6
    ctx.matrix_free(m)


@pytest.mark.parametrize("tokens,rows,cols", [(1, 9728, 2560), (1, 8192, 2048), (1, 7120, 512), (2, 9728, 2560), (2, 16, 512), (2, 6144, 2048)])
def test_activating_product_with_more_tile_pairs_than_blocks(ctx, tokens, rows, cols):
    dev = torch.device("cuda:0")
    (mg, wg), (mu, wu) = (_matrix(ctx, Q.GGML_Q4_K, rows, cols, s) for s in (14, 15))
    x = torch.from_numpy(G.normal(16, tokens, cols).astype(np.float32)).to(dev)
    act = torch.empty(tokens, rows, device=dev)
    torch.cuda.synchronize()
    ctx.matmul_fused_device(Context._parts([(mg, 0, rows), (mu, 0, rows)]), 2, tokens, act, x=x, activate=True)
    ctx.synchronize()
    x64 = x.cpu().numpy().astype(np.float64)
    g, u = x64 @ wg.T, x64 @ wu.T
    assert rel_l2(act.cpu().numpy(), g / (1.0 + np.exp(-g)) * u) <= 5e-6
    ctx.matrix_free(mg)
    ctx.matrix_free(mu)


def test_experts_read_what_the_caller_wrote_behind_the_route():
    """The caller's own kernels write x between the route and the products, on one stream; and the
    two in one call: the same bits as with everything in place beforehand."""
    from gufo_npu_b200 import _capi
    dev = torch.device("cuda:0")
    tokens, k, hidden, ffn, experts = 4, 8, 2048, 512, 16
    stream = torch.cuda.Stream()
    own = Context(0, stream.cuda_stream)
    bank = _capi.ExpertBank(*[_matrix(own, Q.GGML_Q4_K, rows * experts, cols, seed)[0]
                              for seed, rows, cols in ((1, ffn, hidden), (2, ffn, hidden), (3, hidden, ffn))],
                            experts, ffn, hidden)
    gen = torch.Generator(device=dev).manual_seed(3)
    rounds = 24
    logits, xs = (torch.randn(rounds, tokens, w, device=dev, generator=gen) for w in (experts + 1, hidden))
    shared = torch.randn(tokens, hidden, device=dev, generator=gen)
    chosen, weights = torch.empty(tokens, k, dtype=torch.int32, device=dev), torch.empty(tokens, k, device=dev)
    scale = torch.empty(tokens, device=dev)
    buf, act, eo = (torch.empty(tokens * k, w, device=dev) for w in (2 * ffn, ffn, hidden))
    got, one, want = (torch.empty(rounds, tokens, hidden, device=dev) for _ in range(3))
    x = torch.zeros(tokens, hidden, device=dev)
    torch.cuda.synchronize()

    def experts_of(x, out):
        own.moe_ffn_device(bank, chosen, weights, scale, tokens, k, x, hidden, shared, buf, act, eo, out)
    with torch.cuda.stream(stream):
        for r in range(rounds):
            own.route_device(logits[r], experts + 1, tokens, experts, k, chosen, weights, scale)
            stream.synchronize()
            experts_of(xs[r], want[r])
        for r in range(rounds):
            own.route_device(logits[r], experts + 1, tokens, experts, k, chosen, weights, scale)
            torch.mul(xs[r], 1.0, out=x)
            experts_of(x, got[r])
            x.zero_()
        for r in range(rounds):
            torch.mul(xs[r], 1.0, out=x)
            own.moe_layer_device(bank, logits[r], experts + 1, tokens, k, chosen, weights, scale, x, hidden, shared, buf,
                                 act, eo, one[r])
            x.zero_()
    stream.synchronize()
    assert torch.equal(got, want) and torch.equal(one, want)
    own.close()


@pytest.mark.parametrize("tokens,k,hidden,ffn,experts", [(1, 1, 256, 256, 4), (3, 3, 1280, 768, 7), (5, 8, 2048, 512, 16),
                                                         (16, 4, 1536, 256, 64)])
def test_mixture_of_given_experts(ctx, tokens, k, hidden, ffn, experts):
    """The FFN of chosen experts and their weighted sum, with experts left out and chosen twice, one
    to three blocks a row and one to several tiles a thread block, in float64."""
    from gufo_npu_b200 import _capi
    dev = torch.device("cuda:0")
    mats, w = [], []
    for seed, rows, cols in ((1, ffn, hidden), (2, ffn, hidden), (3, hidden, ffn)):
        m, v = _matrix(ctx, Q.GGML_Q4_K, rows * experts, cols, seed)
        mats.append(m)
        w.append(v.reshape(experts, rows, cols))
    bank = _capi.ExpertBank(*mats, experts, ffn, hidden)
    rng = np.random.default_rng(tokens)
    ids = rng.integers(0, experts, (tokens, k)).astype(np.int32)
    if k > 1:
        ids[0, 1] = -1
        ids[-1, 0] = ids[-1, k - 1]
    wt, sc = rng.random((tokens, k)).astype(np.float32), rng.random(tokens).astype(np.float32)
    x, shared = (G.normal(s, tokens, hidden).astype(np.float32) for s in (4, 5))
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    t_ids, t_wt, t_sc, t_x, t_sh = map(up, (ids, wt, sc, x, shared))
    nan = lambda *s: torch.full(s, float("nan"), device=dev)
    buf, act, eo = nan(tokens * k, 2 * ffn), nan(tokens * k, ffn), nan(tokens, k, hidden)
    torch.cuda.synchronize()
    ctx.moe_ffn_device(bank, t_ids, t_wt, t_sc, tokens, k, t_x, hidden, t_sh, buf, act, eo, t_sh)
    ctx.synchronize()
    want = shared.astype(np.float64) * sc[:, None]
    for t in range(tokens):
        for s in range(k):
            e = ids[t, s]
            if e >= 0:
                g, u = w[0][e] @ x[t], w[1][e] @ x[t]
                want[t] += float(wt[t, s]) * (w[2][e] @ (g / (1 + np.exp(-g)) * u))
    assert rel_l2(t_sh.cpu().numpy(), want) <= 5e-6
    # The down rows by themselves, from the activated inputs the call has left: as close as fp32
    # products (3e-7; with 24 bits of the inputs 1e-6 to 3e-6).
    want = shared.astype(np.float64) * sc[:, None]
    for t in range(tokens):
        for s in range(k):
            if ids[t, s] >= 0:
                want[t] += float(wt[t, s]) * (w[2][ids[t, s]] @ act[t * k + s].cpu().numpy().astype(np.float64))
    assert rel_l2(t_sh.cpu().numpy(), want) <= 7e-7
    for m in mats:
        ctx.matrix_free(m)


@pytest.mark.parametrize("ggml_type", [Q.GGML_Q5_K, Q.GGML_Q8_0])
@pytest.mark.parametrize("held", [False, True])
@pytest.mark.parametrize("rows,cols", [(5, 256), (1024, 2304), (3001, 1280), (5999, 256), (5501, 2560), (7301, 512),
                                       (7301, 5376), (2001, 5376)])
def test_split_rows_over_many_groups(ctx, ggml_type, held, rows, cols):
    """Q5_K and Q8_0 rows in two parts: groups of four rows past the end and across the parts, more
    groups than three rounds of blocks (1332 groups, 1776 for one token of Q8_0) of short and of long
    rows, more than one round and one and a half, warps without a block, one unit a warp and several,
    bytes that are borrowed and bytes that the library holds; against float64 over the dequantized
    rows."""
    gen = torch.Generator("cuda").manual_seed(rows + cols)
    per, size = Q.BLOCK_ELEMENTS[ggml_type], Q.BLOCK_BYTES[ggml_type]
    raw = torch.randint(0, 256, (rows * cols // per, size), device="cuda", generator=gen, dtype=torch.uint8)
    for at in ((0, 2) if ggml_type == Q.GGML_Q5_K else (0,)):
        raw[:, at:at + 2] = (1e-4 * (1.0 + torch.rand(raw.shape[0], device="cuda", generator=gen))).half().view(torch.uint8).reshape(-1, 2)
    torch.cuda.synchronize()
    m = (ctx.matrix_upload(ggml_type, raw.cpu().numpy(), rows, cols) if held else
         ctx.matrix_from_device(ggml_type, raw.data_ptr(), rows, cols))
    w = torch.empty(rows, cols, device="cuda")
    torch.cuda.synchronize()
    ctx.dequantize_device(m, 0, rows, w)
    ctx.synchronize()
    parts = Context._parts([(m, 0, rows), (m, 1, 3)])
    for tokens in (1, 2, 3, 5, 8):
        x = torch.randn(tokens, cols, device="cuda", generator=gen)
        y = torch.full((tokens, rows + 3), 7.0, device="cuda")
        torch.cuda.synchronize()
        ctx.matmul_device(parts, 2, x, tokens, y)
        ctx.synchronize()
        want = x.double() @ w.double().T
        scale = x.double().abs() @ w.double().abs().T   # fp32 sums of cols terms: a few roundings of it
        assert ((y[:, :rows].double() - want).abs() <= 2e-6 * scale).all()
        assert torch.equal(y[:, rows:], y[:, 1:4])
    ctx.matrix_free(m)


@pytest.mark.parametrize("ggml_type", [Q.GGML_Q5_K, Q.GGML_Q8_0])
def test_borrowed_bytes_that_the_kernel_before_writes(ctx, ggml_type):
    """A product's outputs are the borrowed weights of the next one: rows of 524288 values keep the
    first busy long after it has let the second start, which must not have read them by then."""
    rows, cols, wide = 4, 256, 524288
    gen = torch.Generator("cuda").manual_seed(7)
    size = rows * cols // Q.BLOCK_ELEMENTS[ggml_type] * Q.BLOCK_BYTES[ggml_type]
    # Bytes of 1 to 63 are normal floats and halves wherever a word or a scale falls.
    want = torch.randint(1, 64, (size,), device="cuda", generator=gen, dtype=torch.uint8)
    source = torch.zeros(size // 4, wide, device="cuda")
    source[:, 0] = want.view(torch.float32)
    one = torch.zeros(wide, device="cuda")
    one[0] = 1.0
    target = torch.zeros(size // 4, device="cuda")
    x = torch.randn(1, cols, device="cuda", generator=gen)
    w = torch.empty(rows, cols, device="cuda")
    y = torch.empty(5, rows, device="cuda")
    torch.cuda.synchronize()
    writer = Context._parts([(ctx.matrix_from_device(Q.GGML_F32, source.data_ptr(), size // 4, wide), 0, size // 4)])
    m = ctx.matrix_from_device(ggml_type, target.data_ptr(), rows, cols)
    for i in range(5):
        target.zero_()
        torch.cuda.synchronize()
        ctx.matmul_device(writer, 1, one, 1, target)
        ctx.matmul_device(Context._parts([(m, 0, rows)]), 1, x, 1, y[i])
        ctx.synchronize()
    assert torch.equal(target.view(torch.uint8), want)
    ctx.dequantize_device(m, 0, rows, w)
    ctx.synchronize()
    exact = x.double() @ w.double().T
    scale = x.double().abs() @ w.double().abs().T
    assert ((y.double() - exact).abs() <= 2e-6 * scale).all()
    ctx.matrix_free(m)


@pytest.mark.parametrize("rows,cols,tokens", [(601, 2052, 1), (1001, 2052, 1), (2371, 1024, 1), (2371, 1028, 1), (2371, 516, 2),
                                              (2371, 516, 3), (1183, 2048, 8), (8199, 2564, 5), (8199, 2564, 17)])
def test_f32_rows_in_every_form(ctx, rows, cols, tokens):
    """Tiles of two rows in one round of blocks and more, of eight rows of one chunk a warp and more,
    matrices beyond the L2; ragged rows, chunks and tokens, two parts; against float64."""
    gen = torch.Generator("cuda").manual_seed(rows + cols)
    w = torch.randn(rows, cols, device="cuda", generator=gen)
    x = torch.randn(tokens, cols, device="cuda", generator=gen)
    y = torch.full((tokens, rows + 3), 7.0, device="cuda")
    torch.cuda.synchronize()
    m = ctx.matrix_from_device(Q.GGML_F32, w.data_ptr(), rows, cols)
    ctx.matmul_device(Context._parts([(m, 0, rows), (m, 1, 3)]), 2, x, tokens, y)
    ctx.synchronize()
    want = x.double() @ w.double().T
    scale = x.double().abs() @ w.double().abs().T   # fp32 sums of cols terms: a few roundings of it
    assert ((y[:, :rows].double() - want).abs() <= 2e-6 * scale).all()
    assert torch.equal(y[:, rows:], y[:, 1:4])
    ctx.matrix_free(m)
