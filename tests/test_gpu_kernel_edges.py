"""The tensor-core kernels, quantizers and weight encoders at the sizes where a tile, a slice of K, a remainder or a
rule of the dispatch ends.  Oracle: the layer's own reconstruction (bit-exact against the CPU oracle elsewhere) in
float64 or exact integer arithmetic, and torch's IEEE division for everything that is bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# A weight is the sum of two e4m3 halves (relative error 2^-8 at most) or an fp16 product (2^-11), the output is rounded
# to bf16 (2^-9): relative to the result's norm no more than their sum.
TOL = 2.0 ** -8 + 2.0 ** -9


def _layer(N, K, d=8, C=4096, G=None, bias=True, seed=0):
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


def _err(mod, y, q, s):
    ref = (q.double() @ mod.dequantize_weight().double().t()) * s.reshape(-1, 1).double()
    if mod.bias is not None:
        ref = ref + mod.bias.double()
    return float((y.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("kernel,N,K,d,C,G", [
    ("large", 100, 256, 8, 4096, None), ("large", 1000, 1024, 4, 4096, None), ("large", 128, 4096, 8, 256, None),
    ("large", 257, 8192, 8, 4096, None), ("large", 520, 2048, 8, 65536, None),
    ("large_grouped", 100, 512, 4, 81, 64), ("large_grouped", 333, 1024, 4, 2048, 64), ("large_grouped", 129, 4096, 8, 256, 128),
    ("large_grouped", 64, 8192, 4, 64, 64)])
def test_split_k_tile_and_slice_edges(kernel, N, K, d, C, G):
    """One to eight slices of K; token tiles around 16, 256, 272 and 384 tokens.  A row's bytes do not depend on how many
    rows there are, a residual adds like a separate addition, a wider output keeps its other columns."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G)
    mod.set_kernel(kernel)
    q, s = quantize_rows(_x(800, K))
    whole = mod.linear_a8(q, s)
    assert _err(mod, whole, q, s) <= TOL
    for M in (1, 15, 17, 64, 255, 257, 272, 273, 384, 385):
        y = mod.linear_a8(q[:M], s[:M])
        assert torch.equal(y, whole[:M]), M
        res = _x(M, N, seed=5)
        assert torch.equal(mod.linear_a8(q[:M], s[:M], residual=res), y + res), M
        out = torch.full((M, N + 3), 7.0, dtype=torch.bfloat16, device="cuda")
        mod.linear_a8(q[:M], s[:M], out=out[:, :N])
        assert torch.equal(out[:, :N], y) and float(out[:, N:].float().min()) == 7.0, M
    assert mod.device_status() == 0


@pytest.mark.parametrize("first,N,K,d,C,G", [
    (8, 128, 256, 8, 4096, None), (8, 333, 768, 4, 256, None), (8, 6144, 256, 8, 4096, None), (8, 200, 2048, 8, 65536, None),
    (12, 128, 512, 4, 81, 64), (12, 1000, 768, 4, 1024, 64), (12, 6144, 256, 8, 256, 128)])
def test_batched_tiles_and_remainders(first, N, K, d, C, G):
    """The kernels that keep the weights in tensor memory: the width of the tiles, the narrower last one, the number of
    tiles per CTA and the way the output leaves change no byte."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G)
    q, s = quantize_rows(_x(3300, K))
    mod.set_kernel(first)
    whole = mod.linear_a8(q, s)
    assert _err(mod, whole, q, s) <= TOL
    for M in (1, 31, 33, 127, 256, 257, 300, 385, 1000, 2049):
        for which in range(first, first + 4):
            mod.set_kernel(which)
            assert torch.equal(mod.linear_a8(q[:M], s[:M]), whole[:M]), (M, which)
        mod.set_kernel(first)
        res = _x(M, N, seed=5)
        assert torch.equal(mod.linear_a8(q[:M], s[:M], residual=res), whole[:M] + res), M
        out = torch.full((M, N + 5), 7.0, dtype=torch.bfloat16, device="cuda")
        mod.linear_a8(q[:M], s[:M], out=out[:, :N])
        assert torch.equal(out[:, :N], whole[:M]) and float(out[:, N:].float().min()) == 7.0, M
    assert mod.device_status() == 0


@pytest.mark.parametrize("N,K,Ms", [(2000, 2048, (33, 300, 1000, 4100)), (1536, 6144, (33, 200, 1100, 2100)),
                                    (6144, 1040, (321, 700, 5000)), (129, 256, (33, 129, 257))])
def test_recipe_tiles(N, K, Ms):
    """Every tile of the dense 8-bit GEMM, ragged token and row ends.  INT8 sums are exact, so the bytes are those of the
    recipe's arithmetic on them; FP8 sums are fp32 in the tensor cores' order."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, 8, 256, bias=False)
    for mode in ("int8_symmetric", "fp8_e4m3fn"):
        sw = mod.weight_row_scale(mode)
        for M in Ms:
            q, s = quantize_rows(_x(M, K), mode)
            if mode == "int8_symmetric":
                acc = q.double() @ mod.decode_weight_int8(sw).double().t()
                want = ((acc.float() * sw.reshape(1, -1)) * s.reshape(-1, 1)).to(torch.bfloat16)
                assert torch.equal(mod.linear_w8a8_int8(q, s, sw), want), M
            else:
                acc = q.double() @ mod.decode_weight_fp8(sw).double().t()
                want = acc * sw.reshape(1, -1).double() * s.reshape(-1, 1).double()
                y = mod.linear_w8a8_fp8(q, s, sw)
                # fp32 sums of K products, each rounded at most once per addition, then one rounding to bf16
                assert float((y.double() - want).norm() / want.norm()) <= 2.0 ** -9 + K * 2.0 ** -24, M
    assert mod.device_status() == 0


def _encode(z, s, mode):
    v = z.float() / s                                   # a tensor divisor: IEEE division
    if mode == "int8_symmetric":
        return v.clamp(-127, 127).round().to(torch.int8)
    return v.clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)


@pytest.mark.parametrize("K,d,C,G", [(16, 8, 16, None), (1008, 4, 128, None), (1040, 8, 256, None), (3088, 4, 2048, None),
                                     (2048, 4, 1024, 64), (1040, 8, 65536, None)])
def test_weight_bytes_equal_division(K, d, C, G):
    """The 8-bit weight rows around a warp's 1,024 weights, for the layer's own row scales and for odd ones."""
    mod = _layer(37, K, d, C, G)
    w = mod.dequantize_weight()
    for mode, decode in (("int8_symmetric", mod.decode_weight_int8), ("fp8_e4m3fn", mod.decode_weight_fp8)):
        own = mod.weight_row_scale(mode).reshape(-1)
        odd = own * torch.logspace(-3, 3, 37, device="cuda") * 1.000123
        for sw in (own, odd):
            got = decode(sw.reshape(mod.weight_row_scale(mode).shape).contiguous())
            got = got if mode == "int8_symmetric" else got.view(torch.uint8)
            assert torch.equal(got, _encode(w, sw.reshape(-1, 1), mode)), mode


@pytest.mark.parametrize("K,d,C", [(1024, 8, 4096), (2048, 4, 1024), (1024, 8, 65536)])
def test_weight_bytes_of_underflowing_products(K, d, C):
    """Group scales so small that products of codewords underflow bf16: a product that does is a zero, to which the shift of
    +0 is added, so its byte is that of +0; one that is still a subnormal keeps its sign."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from sacq_b200 import PrecomputedPackedVectorCodebookLinear
    from sacq_b200.synthetic import make_payload
    p = make_payload(40, K, vector_dim=d, codebook_size=C, group_size=64, seed=9, iters=1, fit=False)
    p["scales"][:, 0::3] = 2.0 ** -133                   # the smallest bf16
    p["scales"][:, 1::3] = 2.0 ** -130
    mod = PrecomputedPackedVectorCodebookLinear(p, None, "cuda")
    w = mod.dequantize_weight()
    for mode, decode in (("int8_symmetric", mod.decode_weight_int8), ("fp8_e4m3fn", mod.decode_weight_fp8)):
        sw = mod.weight_row_scale(mode)
        got = decode(sw)
        got = got if mode == "int8_symmetric" else got.view(torch.uint8)
        assert torch.equal(got, _encode(w, sw.reshape(-1, 1), mode)), mode


# The significands (24 bits, of row scales in [1, 2)) for which the encoders' quotient of some bf16 weight is not the division's:
# by one ulp, of a quotient that no encoding has a boundary next to (tests/test_host_logic.py finds them).
ODD_ROW_SCALES = (0x3f9cdfab, 0x3fbc49ab, 0x3fd0ab43, 0x3fd2d00f, 0x3fdb4e6b, 0x3fe190f3, 0x3fe241ef, 0x3fe5ae9f, 0x3feb3ca3,
                  0x3ff28673, 0x3ff92863)


def test_weight_bytes_for_any_row_scale():
    """A caller's row scales: the odd ones, small whole numbers (quotients that are exact ties), random significands, each at
    magnitudes where a row's quotients reach from zero to saturation.  Weights: every significand of a bf16 number at 16
    exponents, both signs.  The bytes are those of the division; so are those that the GEMMs make for themselves."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from sacq_b200 import PrecomputedPackedVectorCodebookLinear, pack_indices
    g = torch.Generator().manual_seed(4)
    values = (torch.arange(128, 256) / 128.0).reshape(1, -1) * 2.0 ** torch.arange(-9, 7).reshape(-1, 1)
    values = values.reshape(-1) * torch.tensor([1.0, -1.0]).repeat(1024)
    base = torch.cat([torch.tensor(ODD_ROW_SCALES, dtype=torch.int32).view(torch.float32), torch.arange(1, 16).float(),
                      (0x3f800000 + torch.randint(0, 1 << 23, (230,), generator=g, dtype=torch.int32)).view(torch.float32)])
    sw = torch.cat([base * 2.0 ** -8, base * 2.0 ** -3, base]).cuda()
    N, K = sw.numel(), 2048
    idx = torch.stack([torch.randperm(256, generator=g) for _ in range(N)]).reshape(N, 1, 256)
    payload = dict(format="packed_vector_codebook_v1", codebook=values[torch.randperm(2048, generator=g)].reshape(256, 8).bfloat16(),
                   scales=torch.ones(N, 1).bfloat16(), shift=torch.zeros((), dtype=torch.bfloat16), in_features=K, out_features=N,
                   group_size=K, vector_dim=8, packed_indices=pack_indices(idx, 8), index_bits=8, index_shape=(N, 1, 256))
    mod = PrecomputedPackedVectorCodebookLinear(payload, None, "cuda")
    w = mod.dequantize_weight()
    for mode, decode, linear in (("int8_symmetric", mod.decode_weight_int8, mod.linear_w8a8_int8),
                                 ("fp8_e4m3fn", mod.decode_weight_fp8, mod.linear_w8a8_fp8)):
        rows = sw.reshape(mod.weight_row_scale(mode).shape).contiguous()
        want = _encode(w, sw.reshape(-1, 1), mode)
        got = decode(rows)
        assert torch.equal(got if mode == "int8_symmetric" else got.view(torch.uint8), want), mode
        bytes_of = want.float() if mode == "int8_symmetric" else want.view(torch.float8_e4m3fn).float()
        for M in (32, 300):                              # weight bytes made inside the GEMM, and by a kernel of their own
            k = torch.randperm(K, generator=g)[:M].cuda()
            q = torch.zeros(M, K, device="cuda")
            q[torch.arange(M), k] = 1.0
            q = q.to(torch.int8 if mode == "int8_symmetric" else torch.float8_e4m3fn)
            y = linear(q, torch.ones(M, 1, device="cuda"), rows)
            assert torch.equal(y, (bytes_of[:, k].t() * sw.reshape(1, -1)).to(torch.bfloat16)), (mode, M)
    assert mod.device_status() == 0


@pytest.mark.parametrize("M,K", [(1, 8), (3, 100), (5, 2048), (300, 2056), (2, 6144), (297, 6144), (4, 8200), (1, 40000)])
def test_quantizer_bytes_equal_division(M, K):
    """One to four chunks per thread, a warp or a CTA per row, rows longer than the registers hold."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from sacq_b200 import quantize_rows
    x = _x(M, K)
    x[0, : min(K, 6)] = torch.tensor([0.0, -0.0, 1e-39, -1e-39, 3.3e-38, 2.0 ** -126][: min(K, 6)], dtype=torch.bfloat16)
    x[M - 1] *= 1e-20
    for mode, top in (("int8_symmetric", 127.0), ("fp8_e4m3fn", 448.0)):
        q, s = quantize_rows(x, mode)
        want = x.float().abs().amax(1, keepdim=True) / torch.full((M, 1), top, device="cuda")
        assert torch.equal(s.reshape(-1, 1), want)
        got = q if mode == "int8_symmetric" else q.view(torch.uint8)
        assert torch.equal(got, _encode(x, want, mode)), mode


def test_silu_of_every_bf16_value():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from sacq_b200 import act_quantize_rows, quantize_rows
    a = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).cuda().reshape(-1, 64)
    a = torch.where(torch.isfinite(a), a, torch.zeros_like(a))
    for b in (torch.ones_like(a), torch.full_like(a, -0.37)):
        q, s = act_quantize_rows("silu_mul", a, b)
        q2, s2 = quantize_rows(torch.nn.functional.silu(a) * b)
        assert torch.equal(s, s2) and torch.equal(q.view(torch.uint8), q2.view(torch.uint8))


@pytest.mark.parametrize("N,K,d,C,G", [(2048, 2048, 8, 4096, None), (1000, 1024, 4, 1024, 64), (4096, 1024, 8, 65536, None)])
def test_quantizer_inside_the_call_changes_no_byte(N, K, d, C, G):
    """A call that quantizes on its way (few tokens: inside the GEMM) and the quantizer followed by the GEMM."""
    from sacq_b200 import linear_a8_multi, quantize_rows
    mod, other = _layer(N, K, d, C, G), _layer(N // 2, K, d, C, G, bias=False, seed=1)
    for M in (1, 2, 7, 8, 9, 16, 17, 33, 64, 65, 300):
        x = _x(M, K)
        q, s = quantize_rows(x)
        y = mod.linear_a8(q, s)
        assert torch.equal(mod(x), y), M
        assert _err(mod, y, q, s) <= TOL, M
        qi, si = quantize_rows(x, "int8_symmetric")
        assert torch.equal(mod.forward_int8(x), mod.linear_a8i(qi, si)), M
        both = linear_a8_multi([mod, other], q, s)
        assert torch.equal(both[0], y) and torch.equal(both[1], other.linear_a8(q, s)), M
    assert mod.device_status() == 0 and other.device_status() == 0


@pytest.mark.parametrize("N,K,d,C,G", [(256, 1152, 8, 256, None), (256, 2048, 4, 512, None), (128, 2176, 8, 256, None),
                                       (128, 8192, 8, 256, None), (128, 8320, 8, 256, None), (4800, 512, 4, 128, 64)])
def test_quantizer_beside_the_split_k_kernel(N, K, d, C, G):
    """A forward whose quantizer shares SMs with the GEMM has the bytes of the separate calls: around the numbers of tokens
    and the row lengths where its rows change hands, for rows with a pitch, of zeros, infinities and NaN, FP8 and INT8."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G)
    wide = _x(1028, K + 24)
    wide[3] = 0
    wide[5, 7] = float("inf")
    wide[40, K - 1] = float("nan")
    for x in (wide[:, :K].contiguous(), wide[:, 8:K + 8]):
        for M in (49, 97, 369, 370, 371, 1023, 1024, 1025):
            for forward, gemm, mode in ((mod, mod.linear_a8, "fp8_e4m3fn"), (mod.forward_int8, mod.linear_a8i, "int8_symmetric")):
                y, ref = forward(x[:M]), gemm(*quantize_rows(x[:M], mode))
                assert torch.equal(y.view(torch.int16), ref.view(torch.int16)), (M, mode)
    assert mod.device_status() == 0


@pytest.mark.parametrize("N,K,d,C,G", [(2048, 2048, 8, 4096, None), (4224, 1024, 8, 256, None), (1536, 1536, 4, 64, 64),
                                       (1024, 2176, 8, 256, None), (2048, 6144, 8, 256, None)])
def test_rows_per_cta_of_the_quantizer_beside_the_split_k_kernel(N, K, d, C, G):
    """The numbers of tokens at which that quantizer takes a row per CTA or per warp, or leaves the rows to another one."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G)
    x = _x(372, K)
    for M in (52, 64, 65, 100, 255, 256, 257, 298, 299, 340, 341, 372):
        for forward, gemm, mode in ((mod, mod.linear_a8, "fp8_e4m3fn"), (mod.forward_int8, mod.linear_a8i, "int8_symmetric")):
            assert torch.equal(forward(x[:M]), gemm(*quantize_rows(x[:M], mode))), (M, mode)
    assert mod.device_status() == 0


@pytest.mark.parametrize("N,K,d,C", [(6144, 2048, 8, 4096), (4100, 1024, 8, 256), (6200, 512, 8, 256), (1000, 1024, 4, 4096),
                                     (2048, 2048, 8, 65536), (4096, 1536, 8, 65536)])
def test_quantizer_inside_the_split_k_kernel(N, K, d, C):
    """Expander warps that quantize their tokens themselves give the bytes of the separate calls: one or two tokens a warp, tiles
    that end early, rows with a pitch, of zeros, infinities and NaN, a residual, a capture.  It is one launch up to 16 tokens, two
    from 65 on; captured, two where the layer's CTAs wait for SMs."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C)
    mod.set_kernel("large")
    count = mod._lib.sacq_launch_count
    wide = _x(66, K + 16)
    wide[3] = 0
    wide[5, 7] = float("inf")
    wide[9, K - 1] = float("nan")
    res = _x(66, N, seed=4)
    for x in (wide[:, :K].contiguous(), wide[:, 8:K + 8]):
        for M in (1, 2, 8, 15, 16, 17, 31, 32, 33, 48, 64, 65):
            q, s = quantize_rows(x[:M])
            before = count()
            got = mod(x[:M]), mod.forward_residual(x[:M], res[:M])
            launches = count() - before
            assert launches == (2 if M <= 16 else 4 if M == 65 else launches), M
            for y, ref in zip(got, (mod.linear_a8(q, s), mod.linear_a8(q, s, residual=res[:M]))):
                assert torch.equal(y.view(torch.int16), ref.view(torch.int16)), M
    x, stream = wide[:16, :K].contiguous(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    before = count()
    with torch.cuda.graph(graph, stream=stream):
        y = mod(x)
    assert count() - before == (2 if (N, C) == (6144, 4096) else 1)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y.view(torch.int16), mod(x).view(torch.int16)) and mod.device_status() == 0


@pytest.mark.parametrize("N", [1024, 1000])
def test_host_result_stored_by_the_gemm(N):
    """Pinned results: stored by the GEMM where the rows are whole cache lines, copied otherwise."""
    mod = _layer(N, 1024)
    for M in (1, 16, 17, 64, 200):
        x = _x(M, 1024)
        out = torch.full((M, N), 5.0, dtype=torch.bfloat16).pin_memory()
        mod.forward_host(x.cpu().pin_memory(), out)
        torch.cuda.synchronize()
        assert torch.equal(out, mod(x).cpu()), M


@pytest.mark.parametrize("N,K,d,C,G", [(520, 1024, 4, 512, 32), (300, 1536, 8, 4096, 128), (129, 6144, 4, 64, 64), (2048, 2048, 4, 1024, 64)])
def test_unpacked_kernel_token_chunks(N, K, d, C, G):
    """One to six chunks of 16 tokens, up to three of them in a CTA: a token's bytes are those of a call of its own chunk,
    with and without a residual, and columns beyond the layer stay untouched."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G)
    mod.set_kernel("small_mma_unpacked")
    q, s = quantize_rows(_x(96, K))
    whole = torch.cat([mod.linear_a8(q[m:m + 16], s[m:m + 16]) for m in range(0, 96, 16)])
    assert _err(mod, whole, q, s) <= TOL
    for M in (1, 9, 16, 17, 25, 32, 33, 47, 48, 49, 81, 96):
        y = mod.linear_a8(q[:M], s[:M])
        assert torch.equal(y, whole[:M]), M
        res = _x(M, N, seed=5)
        assert torch.equal(mod.linear_a8(q[:M], s[:M], residual=res), y + res), M
        out = torch.full((M, N + 3), 7.0, dtype=torch.bfloat16, device="cuda")
        mod.linear_a8(q[:M], s[:M], out=out[:, :N])
        assert torch.equal(out[:, :N], y) and float(out[:, N:].float().min()) == 7.0, M
    assert mod.device_status() == 0


@pytest.mark.parametrize("N,K,d,C,bits", [(1000, 32, 4, 8192, 16), (16411, 32, 4, 4096, 16), (520, 64, 4, 256, 8), (16411, 64, 8, 4096, 16)])
def test_unpacked_kernel_fewest_warps(N, K, d, C, bits):
    """Layers of one or two MMA steps run CTAs of one or two warps: fewer threads than a CTA has tokens or row biases."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from sacq_b200 import PrecomputedPackedVectorCodebookLinear, pack_indices, quantize_rows
    from sacq_b200.synthetic import make_payload
    p = make_payload(N, K, vector_dim=d, codebook_size=C, group_size=32, seed=N + K, iters=1, fit=False, packed=False)
    idx = p.pop("indices")
    p.update(packed_indices=pack_indices(idx, bits), index_bits=bits, index_shape=tuple(idx.shape))
    bias = torch.randn(N, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
    mod = PrecomputedPackedVectorCodebookLinear(p, bias, "cuda")
    mod.set_kernel("small_mma_unpacked")
    q, s = quantize_rows(_x(64, K))
    for M in (1, 16, 31, 33, 48, 64):
        y = mod.linear_a8(q[:M], s[:M])
        assert _err(mod, y, q[:M], s[:M]) <= TOL, M
    assert mod.device_status() == 0


@pytest.mark.parametrize("kernel,N,K,d,C,G", [
    ("large", 300, 1024, 8, 4096, None), ("large", 129, 4096, 4, 256, None), ("large", 100, 8192, 8, 4096, None),
    ("large_grouped", 300, 2048, 4, 1024, 64), ("large_grouped", 129, 6144, 4, 64, 64)])
def test_split_k_partial_sums(kernel, N, K, d, C, G):
    """Token counts around the widths up to which a cluster's partial sums are sent to their owner and beyond which they are
    fetched, and around the owners' shares: no byte depends on the way."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G)
    mod.set_kernel(kernel)
    q, s = quantize_rows(_x(240, K))
    whole = mod.linear_a8(q, s)
    assert _err(mod, whole, q, s) <= TOL
    for M in (1, 7, 8, 9, 16, 31, 33, 48, 63, 65, 80, 95, 96, 97, 111, 112, 113, 200):
        assert torch.equal(mod.linear_a8(q[:M], s[:M]), whole[:M]), M
    assert mod.device_status() == 0


@pytest.mark.parametrize("N,K,d,C,G,Ms", [(6144, 1152, 8, 65536, None, (289, 305, 320)), (2048, 4224, 4, 16, 64, (768, 700)),
                                          (6144, 1152, 8, 65536, 128, (300, 384))])
def test_split_k_unequal_slices(N, K, d, C, G, Ms):
    """Slices of K of four and five (eight and nine) stages, where the longer one has a box of indices more: the partial sums
    of the others take the place that this box was copied to."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G)
    for M in Ms:
        q, s = quantize_rows(_x(M, K))
        y = mod.linear_a8(q, s)
        assert _err(mod, y, q, s) <= TOL, M
        for _ in range(20):
            assert torch.equal(mod.linear_a8(q, s), y), M
    assert mod.device_status() == 0


@pytest.mark.parametrize("kernel,N,K,d,C,G", [
    ("large_grouped", 200, 29696, 4, 32768, None), ("large_grouped", 300, 28672, 4, 2048, 64), ("large", 300, 28672, 8, 4096, None),
    ("large_grouped", 129, 14336, 4, 4096, 64)])
def test_split_k_deep_layers(kernel, N, K, d, C, G):
    """Layers whose packed indices leave room for a token tile only as they are, without the rest of a 64-byte box: they stay on
    the kernel, with the same widths of tiles, and no byte depends on the width of the boxes."""
    from sacq_b200 import quantize_rows
    mod = _layer(N, K, d, C, G, bias=False)
    assert mod.kernel_for(100) == kernel
    mod.set_kernel(kernel)
    q, s = quantize_rows(_x(400, K))
    whole = mod.linear_a8(q, s)
    assert _err(mod, whole, q, s) <= TOL
    for M in (1, 16, 17, 100, 128, 130, 144, 145, 256, 257, 280, 289, 352, 353, 384):
        assert torch.equal(mod.linear_a8(q[:M], s[:M]), whole[:M]), M
    sw = mod.weight_row_scale("int8_symmetric")          # weight bytes made inside the GEMM: int32 sums are exact
    qi, si = quantize_rows(_x(32, K), "int8_symmetric")
    acc = qi.double() @ mod.decode_weight_int8(sw).double().t()
    want = ((acc.float() * sw.reshape(1, -1)) * si.reshape(-1, 1)).to(torch.bfloat16)
    for M in (1, 16, 32):
        assert torch.equal(mod.linear_w8a8_int8(qi[:M], si[:M], sw), want[:M]), M
    assert mod.device_status() == 0


@pytest.mark.parametrize("N,K,d,C", [(4096, 1024, 8, 256), (6144, 2048, 8, 4096), (4104, 3840, 8, 256), (4096, 2048, 4, 4096),
                                     (4160, 512, 8, 256)])
def test_wide_layers_have_one_order_of_sums(N, K, d, C):
    """A token's outputs are the same bytes in every call of 33 to 959 tokens: alone, in a batch, in the pieces of a chunked call, on
    the rows of a shard; and layers of any widths share a launch."""
    from sacq_b200 import linear_a8_multi, quantize_rows, PrecomputedPackedVectorCodebookLinear
    from sacq_b200.column_parallel import shard_payload
    from sacq_b200.synthetic import make_payload
    p = make_payload(N, K, vector_dim=d, codebook_size=C, seed=N + K, device="cuda", iters=1, fit=False)
    mod = PrecomputedPackedVectorCodebookLinear(p, None, "cuda")
    half = PrecomputedPackedVectorCodebookLinear(shard_payload(p, 1, 2), None, "cuda")
    q, s = quantize_rows(_x(959, K))
    whole = mod.linear_a8(q, s)
    assert _err(mod, whole, q, s) <= TOL
    for M in (33, 100, 255, 256, 257, 300, 319, 320, 385, 513, 559, 560, 561, 700, 958):
        assert torch.equal(mod.linear_a8(q[:M], s[:M]), whole[:M]), M
        assert torch.equal(half.linear_a8(q[:M], s[:M]), whole[:M, N // 2:]), M
    for lo, hi in ((100, 200), (200, 300), (300, 959)):
        assert torch.equal(mod.linear_a8(q[lo:hi], s[lo:hi]), whole[lo:hi]), (lo, hi)
    before = mod._lib.sacq_launch_count()
    both = linear_a8_multi([mod, half], q[:300], s[:300])
    assert mod._lib.sacq_launch_count() - before == 1
    assert torch.equal(both[0], whole[:300]) and torch.equal(both[1], whole[:300, N // 2:])
    assert mod.device_status() == 0 and half.device_status() == 0


@pytest.mark.parametrize("N,K,d,C,G", [(6144, 2048, 8, 4096, None), (4096, 1024, 8, 256, None), (2048, 1024, 8, 65536, None),
                                       (6144, 1536, 4, 4096, None), (6144, 2048, 4, 1024, 64), (4096, 1024, 4, 64, 64),
                                       (2048, 6144, 4, 1024, 64)])
def test_a_shard_gives_the_bytes_of_the_whole_layer(N, K, d, C, G):
    """Told of the whole layer, its rows run the kernel that the layer would, at every number of tokens where a rule looks at the
    width: FP8 and INT8 activations, quantized before or inside the call."""
    from sacq_b200 import quantize_rows, PrecomputedPackedVectorCodebookLinear
    from sacq_b200._lib import SacqError
    from sacq_b200.column_parallel import shard_payload
    from sacq_b200.synthetic import make_payload
    p = make_payload(N, K, vector_dim=d, codebook_size=C, group_size=G, seed=N + K, device="cuda", iters=1, fit=False)
    mod = PrecomputedPackedVectorCodebookLinear(p, None, "cuda")
    x = _x(1030, K)
    sizes = (1, 8, 9, 16, 17, 28, 29, 32, 33, 40, 47, 48, 50, 95, 96, 384, 448, 600, 959, 960, 1023, 1025)
    want = {M: (mod(x[:M]), mod.forward_int8(x[:M])) for M in sizes}
    for rank, world in ((1, 2), (2, 4), (7, 8)):
        part = PrecomputedPackedVectorCodebookLinear(shard_payload(p, rank, world), None, "cuda")
        part.set_shard_of(N)
        cols = slice(rank * N // world, (rank + 1) * N // world)
        for M in sizes:
            assert part.kernel_for(M) == mod.kernel_for(M)
            assert torch.equal(part(x[:M]), want[M][0][:, cols]), (world, M)
            assert torch.equal(part.linear_a8(*quantize_rows(x[:M])), want[M][0][:, cols]), (world, M)
            assert torch.equal(part.forward_int8(x[:M]), want[M][1][:, cols]), (world, M)
        with pytest.raises(SacqError):
            part.set_shard_of(N // world - 1)
        assert part.device_status() == 0
