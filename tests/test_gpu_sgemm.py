"""fp32 GEMM on the tensor cores (csrc/kernels/sgemm.cu) against float64."""
import os
import subprocess
import sys

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


@pytest.mark.parametrize("M,N,K", [(1, 1, 2), (63, 65, 15), (64, 64, 16), (65, 200, 17), (64, 64, 31), (1, 5000, 32), (300, 70, 33),
                                   (2048, 2048, 32), (2048, 2050, 32), (2049, 2500, 16), (2047, 2049, 33)])
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
def test_sgemm_of_short_reductions(M, N, K, ta, tb):
    """Both sides of the lines between the CUDA-core kernels (a rounding per step) and the tensor-core one."""
    a, b, A, B = _operands(M, N, K, ta, tb, 8)
    ref, mag = A.double() @ B.double(), A.double().abs() @ B.double().abs()
    bound = (max(K, 2 * 5 + 1) + 2) * 2.0 ** -24 * mag
    out = C.sgemm(a, b, ta, tb)
    assert bool(((out.double() - ref).abs() <= bound).all())
    acc = torch.ones_like(out)
    C.sgemm(a, b, ta, tb, out=acc, accumulate=True)
    assert torch.equal(acc, out + 1)
    assert C.status_read(True) == 0


def test_sgemm_exact_on_small_integers_and_repeatable():
    g = torch.Generator(device=DEV).manual_seed(2)
    a = torch.randint(-64, 65, (200, 300), device=DEV, generator=g).float()
    b = torch.randint(-64, 65, (300, 140), device=DEV, generator=g).float()
    out = C.sgemm(a, b, False, False)
    assert torch.equal(out, (a.double() @ b.double()).float())
    x, y = torch.randn(128, 4096, device=DEV, generator=g), torch.randn(4096, 128, device=DEV, generator=g)
    assert torch.equal(C.sgemm(x, y), C.sgemm(x, y))


# ------------------------------------------------------------------ the whole fp32 range
# one tile, ragged and unaligned, a reduction split over a cluster, several tiles and chunks
RANGE_SHAPES = [(128, 128, 64), (70, 45, 33), (64, 128, 5000), (130, 260, 192)]
LAYOUTS = [(False, False), (False, True), (True, False), (True, True)]
FMAX, INF, NAN = torch.finfo(torch.float32).max, float("inf"), float("nan")


def _check(a, b, ta, tb):
    """Against float64, whose range holds every fp32 product and sum: infinities and NaNs in the same places, the rest within
    the bound of test_sgemm_against_float64, half of the smallest fp32 number for each rounding, and 2^-148 for each operand
    below 2^-125: 2^-149 for its third part, twice 2^-150 for the products that are left out (second part at most 2^-134,
    third at most 2^-142, against 2^-16 and 2^-8 of the other operand)."""
    A, B = (a.t() if ta else a).double(), (b.t() if tb else b).double()
    K = A.shape[1]
    ref, mag = A @ B, A.abs() @ B.abs()
    out = C.sgemm(a, b, ta, tb)
    assert C.status_read(True) == 0
    over = torch.isfinite(ref) & (ref.abs() > FMAX)
    assert torch.equal(torch.isnan(out), torch.isnan(ref))
    assert torch.equal(out[torch.isinf(ref)], ref[torch.isinf(ref)].float())
    fin = torch.isfinite(ref) & ~over
    small = [(x.abs() < 2.0 ** -125).double() for x in (A, B)]
    bound = (2 * 5 + (K + 63) // 64 + 2) * 2.0 ** -24 * mag + (K + 1) * 2.0 ** -150
    bound += 1.01 * 2.0 ** -148 * (small[0] @ B.abs().nan_to_num(posinf=0) + A.abs().nan_to_num(posinf=0) @ small[1])
    assert bool(((out.double() - ref).abs()[fin] <= bound[fin]).all())
    start = torch.ones_like(out)
    C.sgemm(a, b, ta, tb, out=start, accumulate=True)
    assert bool(((start == out + 1) | (torch.isnan(start) & torch.isnan(out))).all())
    return out


@pytest.mark.parametrize("M,N,K", RANGE_SHAPES)
@pytest.mark.parametrize("ta,tb", LAYOUTS)
@pytest.mark.parametrize("value", [-FMAX, FMAX, 3.3961776e38, INF, -INF, NAN])
def test_sgemm_largest_and_non_finite_operands(M, N, K, ta, tb, value):
    """One such value in A (a mask's lowest value, say) against small, zero and like values in B."""
    a, b, A, B = _operands(M, N, K, ta, tb, 3)
    b.mul_(1e-3)
    A[5, 7] = value
    B[7, 3] = 0.0
    if value in (INF, -INF):
        B[7, 4] = value
        B[9, 6] = value
    out = _check(a, b, ta, tb)
    assert torch.isfinite(out[:5, :3]).all()


@pytest.mark.parametrize("ta,tb", LAYOUTS)
def test_sgemm_largest_operand_on_the_right(ta, tb):
    a, b, A, B = _operands(100, 300, 200, ta, tb, 4)
    a.mul_(1e-3)
    B[150, 129] = -FMAX
    B[3, 299] = INF
    _check(a, b, ta, tb)
    a.fill_(2.0 ** -100)
    b.fill_(FMAX)
    _check(a, b, ta, tb)


def test_sgemm_sums_near_the_largest_number():
    """Parts of a product that are summed apart must not overflow where the sum does not."""
    a = torch.full((128, 64), 2.0 ** 60, device=DEV)
    b = torch.full((64, 128), 2.0 ** 61 * (2 - 2.0 ** -23), device=DEV)   # 64 equal terms: the sum is just under 2^128
    b.mul_(0.99 + 0.01 * torch.rand(64, 128, device=DEV, generator=torch.Generator(device=DEV).manual_seed(5)))
    out = _check(a, b, False, False)
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("M,N,K", RANGE_SHAPES)
@pytest.mark.parametrize("ta,tb", [(False, False), (True, True)])
@pytest.mark.parametrize("exponent", [-100, -110, -115, -120, -126, -135, -149])
def test_sgemm_small_operands_keep_their_bits(M, N, K, ta, tb, exponent):
    """Down to the subnormal numbers of A (which hold fewer bits themselves), against ordinary and against large values."""
    for scale in (1.0, 2.0 ** 100):
        a, b, A, B = _operands(M, N, K, ta, tb, 6)
        a.mul_(2.0 ** (exponent / 2)).mul_(2.0 ** (exponent - exponent / 2))
        b.mul_(scale)
        _check(a, b, ta, tb)
        _check(b.t().contiguous(), a.t().contiguous(), tb, ta)   # the small operand on the right


def test_sgemm_non_finite_operands_in_late_tiles():
    """More tiles per CTA (33) than the mask of left-out pieces has bits."""
    M = N = 69 * 128
    a, b, A, B = _operands(M, N, 33, False, True, 7)
    A[5, 1] = INF
    A[68 * 128 + 5, 1] = -INF
    A[68 * 128 + 70, 0] = NAN
    B[2, 68 * 128 + 100] = INF
    _check(a, b, False, True)


def test_sgemm_as_first_kernel_in_a_capture():
    """A program may capture before it has run any kernel of the library."""
    code = """
import torch
from tinyinfinitrain_b200._lib import C
a, b = torch.randn(128, 64, device="cuda"), torch.randn(64, 96, device="cuda")
out = torch.zeros(128, 96, device="cuda")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    C.sgemm(a, b, False, False, out=out)
graph.replay()
torch.cuda.synchronize()
assert (out.double() - a.double() @ b.double()).abs().max().item() < 1e-4
assert C.status_read(True) == 0
"""
    run = subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
