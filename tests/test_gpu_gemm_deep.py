"""D += A B^T with a long K and few tiles (narrow tiles, deep ring): tile and K tails, strides,
against a float32 product of the same bf16 operands; and the same bits twice (needs a B200).

Bar: float32 accumulation of K products in chains of at most K/16 partial sums, each within 2^-23 of
the sum of magnitudes: K/16 * 2^-23 of sum |a b|, doubled for the tensor core's unrounded inner sums."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(64, 216, 12288), (128, 3456, 1536), (8, 1728, 3840), (64, 64, 256), (130, 70, 264),
                                   (1, 1, 320), (64, 1728, 1000)])
def test_narrow_deep_gemm(M, N, K):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from water_flow_simulation_b200 import _native as nat
    lib = nat.load()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    lda, ldb, ldd = K + 8, K + 16, N + 3
    A = torch.randn(M, lda, device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn(N, ldb, device="cuda", generator=g).to(torch.bfloat16)
    D0 = torch.randn(M, ldd, device="cuda", generator=g)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = []
    for _ in range(2):
        D = D0.clone()
        nat.check(lib.lbm_gemm_bf16(A.data_ptr(), lda, B.data_ptr(), ldb, M, N, K, D.data_ptr(), ldd, 1, None,
                                    err.data_ptr(), torch.cuda.current_stream().cuda_stream), "lbm_gemm_bf16")
        outs.append(D)
    assert int(err.item()) == 0 and torch.equal(*outs)
    a, b = A[:, :K].double(), B[:, :K].double()
    want = D0[:, :N].double() + a @ b.T
    bar = 2 * K / 16 * 2.0 ** -23 * (a.abs() @ b.abs().T) + 2.0 ** -22 * want.abs()
    assert bool(((outs[0][:, :N].double() - want).abs() <= bar).all())
    assert torch.equal(outs[0][:, N:], D0[:, N:])
