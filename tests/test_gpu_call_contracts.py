"""What a call has to keep whichever kernel it runs on: the kernel that was asked for, the precision of its operands, the
order of the stream, the errors it raises.  Oracle: float64 sums of the payload's own codewords and scales."""
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
