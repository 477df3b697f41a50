"""What a call has to keep whichever kernel it runs on: the kernel that was asked for, the precision of its operands, the
order of the stream, the errors it raises.  Oracle: float64 sums of the payload's own codewords and scales."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(N, K, d=8, C=4096, G=None, bias=False, seed=0):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from sacq_b200 import PrecomputedPackedVectorCodebookLinear
    from sacq_b200.synthetic import make_payload
    p = make_payload(N, K, vector_dim=d, codebook_size=C, group_size=G, seed=N + K + C + seed, device="cuda", iters=1, fit=False)
    b = (torch.randn(N, generator=torch.Generator().manual_seed(1)) * 0.05).to(torch.bfloat16) if bias else None
    return PrecomputedPackedVectorCodebookLinear(p, b, "cuda")


def _x(M, K, seed=3):
    from sacq_b200.synthetic import make_activations
    return make_activations(M, K, seed=seed).cuda()


@pytest.mark.parametrize("N,K,M", [(2048, 2048, 41), (1024, 6144, 20), (3000, 3072, 47)])
def test_a_forced_kernel_is_the_one_that_runs(N, K, M):
    """Grouped scales, where several kernels take the layer.  The index-unpacking kernel sums a token in one order however
    many there are, so a larger call repeats the bytes of a 16-token one; kernel_for() names the kernel whose bytes the
    automatic choice gives."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, 4, 256, 64)
    q, s = quantize_rows(_x(M, K))
    outs = {}
    for which in ("small", "small_mma_unpacked"):
        mod.set_kernel(which)
        outs[which] = mod.linear_a8(q, s)
        assert torch.equal(outs[which][:16], mod.linear_a8(q[:16], s[:16])), which
    mod.set_kernel("auto")
    assert mod.kernel_for(M) == "small" and torch.equal(mod.linear_a8(q, s), outs["small"])
    assert torch.equal(mod(_x(M, K)), outs["small"])


def _exact(mod, q, s):
    """Float64 sums of codeword x scale (not rounded to bf16 as the reconstruction is), rounded once to bf16."""
    bits, n, k, g = mod.index_bits, mod.out_features, mod.in_features, mod.group_size
    planes = (mod.packed_indices[: mod._packed_bytes].unsqueeze(1) >> torch.arange(8, device="cuda", dtype=torch.uint8)) & 1
    fields = planes.reshape(-1)[: n * k // mod.vector_dim * bits].reshape(-1, bits).long()
    w = mod.codebook.double()[(fields << torch.arange(bits, device="cuda")).sum(1)].reshape(n, k // g, g) * mod.scales.double().unsqueeze(-1)
    y = q.double() @ w.reshape(n, k).t() * s.reshape(-1, 1).double()
    return (y if mod.bias is None else y + mod.bias.double()).to(torch.bfloat16)


@pytest.mark.parametrize("N,K,d,C,G", [
    (6144, 1024, 4, 1024, 64), (1000, 1024, 4, 81, 64), (129, 8192, 4, 64, 64), (300, 1536, 8, 4096, 128),   # grouped scales
    (1024, 2048, 8, 4096, None), (264, 1024, 4, 700, None), (520, 2048, 8, 65536, None)])                     # one per row
def test_few_tokens_multiply_exact_weights(N, K, d, C, G):
    """Whatever kernel takes a call of fewer than 96 tokens on grouped scales (48 on layers of 2,048 outputs, 33 on the widest),
    or of fewer than 48 on INT8 activations (any number, where the codebook does not fit shared memory), its weights are
    codeword x scale with all 16 significant bits.
    An fp32 sum of up to 16 x 512 products is within about 2^-19 of the result, so about one output in 2^10 lies close
    enough to the middle between two bf16 values to be rounded the other way; weights of 11 bits put every tenth there."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G, bias=True)
    # rows and groups of very different scale: a row's own largest scale is what its operands are brought to
    mod.scales *= torch.logspace(-9, 3, N, base=2.0, device="cuda").to(torch.bfloat16).unsqueeze(1)
    if G is not None:
        mod.scales[:, ::3] *= 2.0 ** -5
    from sacq_b200 import PrecomputedPackedVectorCodebookLinear
    mod = PrecomputedPackedVectorCodebookLinear(
        {"codebook": mod.codebook, "scales": mod.scales, "in_features": K, "out_features": N, "group_size": G or K, "vector_dim": d,
         "packed_indices": mod.packed_indices[: mod._packed_bytes], "index_bits": mod.index_bits, "index_shape": mod.index_shape},
        mod.bias, "cuda")
    x = _x(300, K)
    for mode, call, sizes in (("fp8_e4m3fn", mod.linear_a8, (1, 17, 32) + ((33, 47, 48, 64, 95) if N < 2048 else ()) if G is not None else (1, 33)),
                              ("int8_symmetric", mod.linear_a8i, (1, 4, 16, 17, 33, 47) + ((48, 95, 300) if C > 4096 else ()))):
        q, s = quantize_rows(x, mode)
        for M in sizes:
            y, want = call(q[:M].contiguous(), s[:M].contiguous()), _exact(mod, q[:M], s[:M])
            assert float((y != want).float().mean()) <= 2.0 ** -8, (mode, M)
            # one step of bf16 is up to 2^-7 of the value: 2^-8 of the outputs off by one are 2^-11 of the norm
            assert float((y.double() - want.double()).norm() / want.double().norm()) <= 2.0 ** -11, (mode, M)
    assert mod.device_status() == 0


@pytest.mark.parametrize("K,d,C,G", [(28672, 4, 4096, None), (30720, 4, 4096, None), (32768, 4, 4096, None),
                                     (28672, 4, 2048, 64), (32768, 4, 2048, 64), (16384, 8, 65536, None)])
def test_deep_layers_run_at_every_token_count(K, d, C, G):
    """Layers whose slice of K leaves little or no shared memory for activation tiles: every token count runs, on e4m3 and
    INT8 activations and on the two recipes, and a forced kernel that can run 16 tokens can run 1,000."""
    from sacq_b200 import quantize_rows
    mod = _layer(64, K, d, C, G)
    w = mod.dequantize_weight().double()
    tol = 2.0 ** -8 + 2.0 ** -9                          # e4m3 halves or bf16 reconstruction, bf16 output
    x = _x(1100, K)
    for mode, call in (("fp8_e4m3fn", mod.linear_a8), ("int8_symmetric", mod.linear_a8i)):
        q, s = quantize_rows(x, mode)
        ref = q.double() @ w.t() * s.double()
        for M in (16, 17, 33, 65, 129, 200, 257, 700, 1000, 1023, 1100):
            y = call(q[:M].contiguous(), s[:M].contiguous()).double()
            assert float((y - ref[:M]).norm() / ref[:M].norm()) <= tol, (mode, M)
    q, s = quantize_rows(x)
    ref = q.double() @ w.t() * s.double()
    for which in ("large", "large_grouped", "large_tmem", "large_tmem_grouped"):
        mod.set_kernel(which)
        try:
            mod.linear_a8(q[:16], s[:16])
        except Exception as e:
            assert getattr(e, "code", 0) == -2, which
            continue
        for M in (385, 700, 1000):
            y = mod.linear_a8(q[:M], s[:M])
            assert float((y.double() - ref[:M]).norm() / ref[:M].norm()) <= tol, (which, M)
            assert torch.equal(y[:16], mod.linear_a8(q[:16], s[:16])), (which, M)
    mod.set_kernel("auto")
    sw = mod.weight_row_scale("int8_symmetric")
    qi, si = quantize_rows(x[:20].contiguous(), "int8_symmetric")
    acc = qi.double() @ mod.decode_weight_int8(sw).double().t()
    assert torch.equal(mod.linear_w8a8_int8(qi, si, sw), ((acc.float() * sw.reshape(1, -1)) * si).to(torch.bfloat16))
    assert mod.device_status() == 0


@pytest.mark.parametrize("mode", ["int8_symmetric", "fp8_e4m3fn"])
def test_recipe_reads_row_scales_of_the_kernel_in_front(mode):
    """The recipe's row scales may be written by the launch directly before the call, on the same stream: here the
    quantizer, which lets the kernel behind it start early, on the layer's own weights."""
    from sacq_b200 import quantize_rows
    mod = _layer(6144, 2048)
    call = mod.linear_w8a8_int8 if mode == "int8_symmetric" else mod.linear_w8a8_fp8
    w = mod.dequantize_weight()
    want_sw = mod.weight_row_scale(mode).clone()
    for M in (1, 16, 200, 1024):                        # inside the GEMM, and as rows of their own
        q, s = quantize_rows(_x(M, 2048), mode)
        want = call(q, s, want_sw)
        wq = torch.empty(6144, 2048, dtype=torch.uint8, device="cuda")
        for _ in range(10):
            sw = torch.full((6144, 1), 1e30, device="cuda")
            quantize_rows(w, mode, out=wq, scale_out=sw)
            assert torch.equal(call(q, s, sw), want), M
            assert torch.equal(sw, want_sw)


@pytest.mark.parametrize("N,K,C,G", [(6144, 256, 1024, 64), (6137, 512, 81, 64)])
def test_staged_output_and_the_next_tiles_activations(N, K, C, G):
    """The persistent kernel for grouped scales stages a wide tile's output where the next tile's activations go.  With a
    residual or an unaligned output its warps read the stage back themselves: many short tiles per CTA, every row compared
    with the same rows of a call that has one tile each."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, 4, C, G)
    mod.set_kernel("large_tmem_grouped")
    M = 3000
    q, s = quantize_rows(_x(M, K))
    parts = torch.cat([mod.linear_a8(q[i:i + 128], s[i:i + 128]) for i in range(0, M, 128)])
    res = _x(M, N, seed=5)
    wide = torch.full((M, N + 3), 7.0, dtype=torch.bfloat16, device="cuda")
    for _ in range(5):
        assert torch.equal(mod.linear_a8(q, s, residual=res), parts + res)
        mod.linear_a8(q, s, out=wide[:, :N])
        assert torch.equal(wide[:, :N], parts)
    assert mod.device_status() == 0


@pytest.mark.parametrize("M,K", [(1, 32776), (3, 102400), (297, 8200), (300, 14336), (512, 40960), (298, 8196), (2, 40001)])
def test_activations_of_wide_rows(M, K):
    """Rows of more chunks than the registers hold, aligned and not: the bytes of the separate tensor operations."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import torch.nn.functional as F
    from sacq_b200 import act_quantize_rows, modulate_quantize_rows, quantize_rows
    a, b = _x(M, K), _x(M, K, seed=4)
    a[M - 1] *= 1e-3
    for got, y in ((act_quantize_rows("silu_mul", a, b), F.silu(a) * b), (act_quantize_rows("gelu", a), F.gelu(a)),
                   (modulate_quantize_rows(a, b[0], b[M - 1]), a * (1 + b[0]) + b[M - 1])):
        want = quantize_rows(y)
        assert torch.equal(got[0].view(torch.uint8), want[0].view(torch.uint8)) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("M,K", [(1, 32776), (3, 51200), (297, 8200), (300, 14336), (298, 8196), (2, 40001)])
def test_layernorm_of_wide_rows(M, K):
    """The same row lengths through the fused LayerNorm: its y within two bf16 steps of torch's in fp32 (another order of
    the sums, and the step of the modulation), its bytes those of its own y."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import torch.nn.functional as F
    from sacq_b200 import layernorm_quantize_rows, quantize_rows
    x, v = _x(M, K), _x(4, K, seed=4)
    for mod in (False, True):
        q, s, y = layernorm_quantize_rows(x, v[0], v[1], 1e-5, *((v[2], v[3]) if mod else ()), return_normalized=True)
        want = F.layer_norm(x.float(), (K,), v[0].float(), v[1].float(), 1e-5).to(torch.bfloat16)
        if mod:
            want = want * (1 + v[2]) + v[3]
        assert float((y.float() - want.float()).norm() / want.float().norm()) <= 2.0 ** -8
        want = quantize_rows(y)
        assert torch.equal(q.view(torch.uint8), want[0].view(torch.uint8)) and torch.equal(s, want[1])


def test_an_allocation_that_fails_raises_out_of_memory():
    """Callers catch torch.OutOfMemoryError, free memory and try again: a RuntimeError of another kind would pass them by.
    The output of 2^23 rows of 2^14 (256 GB) is more than the device has; its input is 1 GB."""
    mod = _layer(1 << 14, 64, 8, 16)
    x = torch.zeros(1 << 23, 64, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(torch.OutOfMemoryError):
        mod(x)
    y = mod(x[:16])                                     # and the layer goes on working
    assert tuple(y.shape) == (16, 1 << 14) and mod.device_status() == 0


@pytest.mark.parametrize("flag,wanted", [(True, True), (1, True), ("yes", True), (False, False), (0, False), (None, False)])
def test_return_normalized_takes_any_truth_value(flag, wanted):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from sacq_b200 import layernorm_quantize_rows
    out = layernorm_quantize_rows(_x(5, 64), return_normalized=flag)
    assert len(out) == (3 if wanted else 2)


def test_strided_inputs_are_read_where_they_lie():
    """A slice of a wider tensor, in two and in three dimensions, allocates its output and nothing else; other layouts are
    made contiguous first.  All give the bytes of the contiguous input."""
    mod = _layer(256, 512)
    wide = _x(6 * 40, 1024).reshape(6, 40, 1024)
    cases = [wide[..., :512], wide[..., 512:], wide[:, 7, :512], wide[0, :, 512:], wide[:3, :, :512].transpose(0, 1),
             _x(512, 40).t(), _x(512, 6).t().unsqueeze(0), wide[..., :512].float()]
    for i, x in enumerate(cases):
        want = mod(x.contiguous())
        torch.cuda.synchronize()
        before = torch.cuda.memory_stats()["allocation.all.allocated"]
        y = mod(x)
        made = torch.cuda.memory_stats()["allocation.all.allocated"] - before
        assert torch.equal(y, want) and y.dtype == x.dtype and tuple(y.shape) == (*x.shape[:-1], 256), i
        assert i >= 4 or made == 1, (i, made)


@pytest.mark.parametrize("N,K,d,C,G", [(300, 960, 4, 256, 64), (129, 576, 4, 256, 64), (1000, 1088, 8, 65536, 64),
                                       (2048, 4160, 4, 256, 64), (64, 64, 4, 256, 64)])
def test_grouped_layers_that_end_inside_a_stage(N, K, d, C, G):
    """K a multiple of 64 but not of 128: the tensor-core kernel takes the layer, to the last group, at every slice count."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G, bias=True)
    w, tol = mod.dequantize_weight().double(), 2.0 ** -8 + 2.0 ** -9
    x = _x(1100, K)
    for mode, call in (("fp8_e4m3fn", mod.linear_a8), ("int8_symmetric", mod.linear_a8i)):
        q, s = quantize_rows(x, mode)
        ref = q.double() @ w.t() * s.double() + mod.bias.double()
        for M in (1, 17, 47, 48, 96, 300, 1024, 1100):
            y = call(q[:M].contiguous(), s[:M].contiguous()).double()
            assert float((y - ref[:M]).norm() / ref[:M].norm()) <= tol, (mode, M)
    assert mod.kernel_for(300) == "large_grouped"
    q, s = quantize_rows(x)
    mod.set_kernel("large_grouped")
    whole = mod.linear_a8(q, s)
    assert torch.equal(mod.linear_a8(q[:20], s[:20]), whole[:20]) and mod.device_status() == 0


@pytest.mark.parametrize("N,K,d,C,G", [(300, 1024, 8, 65536, 128), (64, 32768, 4, 2048, 64)])
def test_grouped_layers_without_a_warp_mma_kernel(N, K, d, C, G):
    """A codebook or a row of indices that the index-unpacking kernel has no room for: the split-K kernel takes the layer
    from one token on, with exact weights."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G, bias=True)
    for M in (1, 5, 16, 40):
        q, s = quantize_rows(_x(M, K))
        y, want = mod.linear_a8(q, s), _exact(mod, q, s)
        assert mod.kernel_for(M) == "large_grouped"
        # sums of up to 32,768 products: four times the bound of the shorter ones
        assert float((y.double() - want.double()).norm() / want.double().norm()) <= 2.0 ** -10, M
        assert torch.equal(mod(_x(M, K)), y)
    assert mod.device_status() == 0


@pytest.mark.parametrize("N,K,d,C,G", [(2048, 2048, 4, 4096, None), (1024, 1024, 4, 256, 64)])
def test_a_captured_call_gives_the_eager_bytes(N, K, d, C, G):
    """An eager call of few tokens quantizes inside the GEMM, a captured one in a launch of its own."""
    mod = _layer(N, K, d, C, G, bias=True)
    for M in (1, 8, 16, 17):
        x = _x(M, K)
        want = mod(x)
        before = mod._lib.sacq_launch_count()
        mod(x)
        eager = mod._lib.sacq_launch_count() - before
        torch.cuda.synchronize()
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            mod(x)                                      # the stream's workspace
        torch.cuda.synchronize()
        before = mod._lib.sacq_launch_count()
        with torch.cuda.graph(graph, stream=stream):
            y = mod(x)
        assert mod._lib.sacq_launch_count() - before >= max(eager, 2), M
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want), M


def test_host_forward_leaves_other_threads_running():
    """A result in pageable memory is copied by a call that waits for the stream: other Python threads run meanwhile.  And
    threads that share a stream each get their own result."""
    import threading
    import time
    mod = _layer(256, 512)
    xs = [_x(40, 512, seed=i).cpu() for i in range(4)]
    want = [mod(x.cuda()).cpu() for x in xs]
    ticks, stop = [0], threading.Event()

    def count():
        while not stop.is_set():
            time.sleep(0.001)
            ticks[0] += 1
    t = threading.Thread(target=count)
    t.start()
    torch.cuda.synchronize()
    torch.cuda._sleep(400_000_000)                      # about 0.2 s of a busy stream
    before = ticks[0]
    y = mod.forward_host(xs[0])
    during = ticks[0] - before
    stop.set()
    t.join()
    torch.cuda.synchronize()
    assert torch.equal(y, want[0]) and during >= 20, during

    bad = []

    def work(i):
        for _ in range(50):
            got = mod.forward_host(xs[i])
            torch.cuda.current_stream().synchronize()
            if not torch.equal(got, want[i]):
                bad.append(i)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("N,K,d,C,G,M", [(256, 1024, 8, 4096, None, 4), (256, 1024, 4, 256, 64, 300), (256, 1024, 8, 4096, None, 300)])
def test_linear_bf16_leaves_the_quantized_activations(N, K, d, C, G, M):
    """The C entry point is the quantizer and the GEMM in turn: its scratch holds what the first wrote."""
    from sacq_b200 import _lib, quantize_rows
    mod = _layer(N, K, d, C, G)
    x = _x(M, K)
    q, s = quantize_rows(x)
    qs, ss = torch.full((M, K), 0x55, dtype=torch.uint8, device="cuda"), torch.full((M,), -1.0, device="cuda")
    y, lib = torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), mod._lib
    ws = torch.zeros(int(lib.sacq_workspace_bytes(mod._handle, M)), dtype=torch.uint8, device="cuda")
    _lib.check(lib.sacq_linear_bf16(mod._handle, x.data_ptr(), K, M, qs.data_ptr(), ss.data_ptr(), y.data_ptr(), N,
                                    ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(y, mod(x)) and torch.equal(qs, q.view(torch.uint8)) and torch.equal(ss, s.reshape(-1))


def test_recipe_takes_more_tokens_than_the_small_tiles_can():
    """8.4 to 16.7 million tokens: more tiles of 128 than a grid has, but not of 256."""
    from sacq_b200 import quantize_rows
    mod = _layer(64, 16, 8, 16)
    M = 65535 * 128 + 77
    sw = mod.weight_row_scale("int8_symmetric")
    q, s = quantize_rows(_x(1 << 12, 16).repeat(M // (1 << 12) + 1, 1)[:M], "int8_symmetric")
    y = mod.linear_w8a8_int8(q, s, sw)
    assert torch.equal(y[-500:], mod.linear_w8a8_int8(q[-500:].contiguous(), s[-500:].contiguous(), sw))


@pytest.mark.parametrize("N,K,d,C,G,M", [(2048, 6144, 8, 4096, None, 64), (6144, 2048, 8, 4096, None, 16), (6144, 2048, 8, 4096, None, 700),
                                         (2048, 2048, 4, 1024, 64, 64), (6144, 2048, 4, 1024, 64, 16), (1536, 1536, 4, 1024, 64, 16)])
def test_a_call_is_cut_up_once(N, K, d, C, G, M):
    """The search for the cut of a split-K call is host time that each call pays, no more than once."""
    from sacq_b200 import _lib, quantize_rows
    mod = _layer(N, K, d, C, G)
    x, res = _x(M, K), _x(M, N, seed=4)
    q, s = quantize_rows(x)
    lib = ctypes.CDLL(_lib.LIB_PATH)
    lib.sacq_split_search_count.restype = ctypes.c_int64
    for call, most in ((lambda: mod(x), 1), (lambda: mod.forward_int8(x), 1), (lambda: mod.forward_residual(x, res), 1),
                       (lambda: mod.linear_a8(q, s), 1)):
        call()
        before = lib.sacq_split_search_count()
        call()
        assert lib.sacq_split_search_count() - before <= most


@pytest.mark.parametrize("N,K,first", [(2048, 6144, 33), (2048, 4096, 33), (4736, 3072, 17), (4096, 1024, 17), (5632, 3072, 9),
                                       (6144, 2048, 9), (6020, 2048, 9), (5000, 2048, 17), (2048, 2048, 48)])
def test_where_the_grouped_split_k_kernel_takes_over(N, K, first):
    """From the first number of tokens at which it is the faster one both for a forward and for a call on quantized activations;
    below, the bytes are the index-unpacking kernel's."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, 4, 1024, 64)
    q, s = quantize_rows(_x(first, K))
    assert mod.kernel_for(first - 1) == "small" and mod.kernel_for(first) == "large_grouped"
    below = mod.linear_a8(q[:first - 1], s[:first - 1])
    mod.set_kernel("small_mma_unpacked")
    assert torch.equal(mod.linear_a8(q[:first - 1], s[:first - 1]), below)


@pytest.mark.parametrize("N,K,kernel", [(6144, 2048, "large"), (6020, 2048, "large"), (4090, 3072, "small"), (4096, 3072, "large"),
                                        (5992, 2048, "small"), (6144, 1536, "small"), (2048, 6144, "small")])
def test_which_layers_leave_the_small_m_kernel_at_one_token(N, K, kernel):
    """Rows count in whole row tiles, so a layer that lacks a few rows of a wider one runs on its kernel."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K)
    q, s = quantize_rows(_x(16, K))
    for M in (1, 16):
        assert mod.kernel_for(M) == kernel
        y = mod.linear_a8(q[:M], s[:M])
        mod.set_kernel(kernel)
        assert torch.equal(mod.linear_a8(q[:M], s[:M]), y)
        mod.set_kernel("auto")
