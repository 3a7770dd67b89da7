"""Dense product with fp32 output (router logits): token tiles of all sizes, ragged rows, columns and
reduction lengths, both layouts of the weights, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows around a tile of 16 and of 128, many tiles; reductions of one k-block (with a tail) up to 112, below and
# above the stages in flight; columns around half a tile, one tile and several
@pytest.mark.parametrize("S,K,N", [(1, 64, 8), (16, 7168, 32), (127, 520, 64), (128, 256, 72), (129, 2048, 128),
                                   (300, 8, 200), (1531, 1024, 256), (40, 4096, 264), (4096, 512, 1000), (20000, 64, 16)])
def test_dense_matches_fp64(S, K, N):
    from moonep_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(S + K + N)
    a = torch.randn(S, K, device="cuda", generator=g).bfloat16()
    b = torch.randn(K, N, device="cuda", generator=g).bfloat16()
    want = a.double() @ b.double()
    # fp32 sums of K exact products: K/2 roundings of at most 2^-24 of the partial sum's size, sqrt(K) here
    bound = 2.0 ** -24 * K * (a.double().abs() @ b.double().abs()) / K ** 0.5 + 1e-30
    for got in (gemm.dense(a, b), gemm.dense(a, b.t().contiguous(), b_is_kn=False)):
        assert got.dtype == torch.float32 and got.shape == (S, N)
        assert bool(((got.double() - want).abs() <= bound).all())
        assert torch.equal(got, gemm.dense(a, b)), "the order of the sums is fixed"
    gemm.check_status()


# more tiles than CTAs: the token-major kernel takes them, with the same sums
@pytest.mark.parametrize("S,K,N", [(4096, 264, 1000), (20000, 512, 264), (2500, 1024, 4104), (40000, 64, 72)])
def test_large_products(S, K, N):
    from moonep_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(S + K + N)
    a = torch.randn(S, K, device="cuda", generator=g).bfloat16()
    b = torch.randn(K, N, device="cuda", generator=g).bfloat16()
    bt = b.t().contiguous()
    want = a.double() @ b.double()
    bound = 2.0 ** -24 * K ** 0.5 * (a.double().abs() @ b.double().abs()) + 1e-30
    got = gemm.dense(a, b)
    assert bool(((got.double() - want).abs() <= bound).all())
    assert torch.equal(gemm.dense(a, bt, b_is_kn=False), got)
    for r in (0, S // 2, S - 100):       # a few of its rows alone fit the other kernel
        assert torch.equal(gemm.dense(a[r:r + 100].contiguous(), b), got[r:r + 100])
    gemm.check_status()


# stages of four and of two k-blocks, the last one partly filled, reductions shorter and longer than the ring
@pytest.mark.parametrize("N", [32, 128])
@pytest.mark.parametrize("S", [5, 1000])
@pytest.mark.parametrize("K", [8, 320, 1480, 5800])
def test_last_stage(S, K, N):
    from moonep_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(S + K + N)
    a = torch.randn(S, K, device="cuda", generator=g).bfloat16()
    b = torch.randn(K, N, device="cuda", generator=g).bfloat16()
    # exact products, K additions that are each off by at most one unit of a running sum below sum |a b|
    bound = 2.0 ** -23 * K * (a.double().abs() @ b.double().abs())
    for got in (gemm.dense(a, b), gemm.dense(a, b.t().contiguous(), b_is_kn=False)):
        assert bool(((got.double() - a.double() @ b.double()).abs() <= bound).all())
    gemm.check_status()
