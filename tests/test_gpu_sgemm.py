"""fp32 GEMM on the tensor cores (csrc/kernels/sgemm.cu) against float64."""
import pytest
import torch

from tinyinfinitrain_b200._lib import C

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _operands(M, N, K, ta, tb, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    a = torch.randn((K, M) if ta else (M, K), device=DEV, generator=g)
    b = torch.randn((N, K) if tb else (K, N), device=DEV, generator=g)
    return a, b, (a.t() if ta else a), (b.t() if tb else b)


# tile and chunk edges, ragged sizes (no 16-byte alignment), one element, cluster splits 2, 4, 8 (few tiles, long K),
# several tiles per CTA (tiles > SMs)
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (128, 128, 64), (129, 127, 65), (70, 45, 33), (130, 260, 192), (128, 768, 3072),
                                   (64, 128, 5000), (3, 1000, 513), (2048, 1300, 100), (1664, 1664, 128)])
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
def test_sgemm_against_float64(M, N, K, ta, tb):
    a, b, A, B = _operands(M, N, K, ta, tb)
    ref = A.double() @ B.double()
    mag = A.double().abs() @ B.double().abs()
    # per element: at most 2^-23 for each truncating addition of a 64-step chunk (24, of which 20 at 2^-8 of the size), 2^-24
    # for each rounding of the chunk sums, 2^-23 for the dropped products and the store
    bound = (2 * 5 + (K + 63) // 64 + 2) * 2.0 ** -24 * mag + 1e-30
    out = C.sgemm(a, b, ta, tb)
    assert bool(((out.double() - ref).abs() <= bound).all())
    acc = torch.ones_like(out)
    C.sgemm(a, b, ta, tb, out=acc, accumulate=True)
    assert bool(((acc.double() - ref - 1).abs() <= bound + 2.0 ** -23 * (ref.abs() + 1)).all())
    assert C.status_read(True) == 0


@pytest.mark.parametrize("M,N,K", [(256, 256, 768), (128, 128, 8192)])
@pytest.mark.parametrize("positive", [False, True])
def test_sgemm_is_as_accurate_as_an_fp32_chain(M, N, K, positive):
    """The rms error stays below that of the sequential fp32 multiply-add chain (one rounding per step)."""
    a, b, A, B = _operands(M, N, K, False, False, 1)
    if positive:   # sums that grow: the case where truncating accumulation would drift
        a, b = a.abs_(), b.abs_()
    ref = A.double() @ B.double()
    chain = torch.zeros(M, N, device=DEV)
    for k in range(K):
        chain = (chain.double() + A[:, k:k + 1].double() * B[k:k + 1].double()).float()   # a fused multiply-add
    err = (C.sgemm(a, b, False, False).double() - ref).norm()
    assert err <= (chain.double() - ref).norm()


def test_sgemm_exact_on_small_integers_and_repeatable():
    g = torch.Generator(device=DEV).manual_seed(2)
    a = torch.randint(-64, 65, (200, 300), device=DEV, generator=g).float()
    b = torch.randint(-64, 65, (300, 140), device=DEV, generator=g).float()
    out = C.sgemm(a, b, False, False)
    assert torch.equal(out, (a.double() @ b.double()).float())
    x, y = torch.randn(128, 4096, device=DEV, generator=g), torch.randn(4096, 128, device=DEV, generator=g)
    assert torch.equal(C.sgemm(x, y), C.sgemm(x, y))
