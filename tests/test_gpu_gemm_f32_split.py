"""The fp32 GEMM's tensor-core path (operands split into three bf16 parts) through cavs_gemm_f32, against a 64-bit product of
the same operands: every way of reading an operand, ragged edges of tiles and k blocks, accumulation, and values that have
no finite split.

Tolerance: the error of a value is at most that of k rounded fp32 additions of its terms, k * 2^-24 * sum |a||b|; the
path keeps within the bound for 8 such additions whatever k is (2^-24 per operand split, 3 sums per 64 values)."""
import ctypes

import pytest
import torch

from cavs_b200 import check, lib

pytestmark = pytest.mark.gpu
ll = ctypes.c_longlong


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _gemm(C, A, B, m, n, k, accumulate=0):
    check(lib().cavs_gemm_f32(_p(C), ll(C.stride(0)), accumulate, _p(A), ll(A.stride(0)), ll(A.stride(1)), _p(B), ll(B.stride(0)),
                              ll(B.stride(1)), m, n, k, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()


def _operand(rows, cols, layout, gen, cuda):
    """layout: "row" contiguous, "pad" with an odd pitch, "col" transposed, "colpad" transposed with an odd pitch."""
    shape = (rows, cols) if layout in ("row", "pad") else (cols, rows)
    pad = 3 if layout.endswith("pad") else 0
    t = torch.randn((shape[0], shape[1] + pad), generator=gen).to(cuda)[:, :shape[1]]
    return t if layout in ("row", "pad") else t.t()


@pytest.mark.parametrize("la", ["row", "pad", "col", "colpad"])
@pytest.mark.parametrize("lb", ["row", "pad", "col", "colpad"])
@pytest.mark.parametrize("m,n,k", [(600, 640, 256), (601, 643, 257), (130, 1996, 1028), (3000, 2100, 68)])
def test_operand_layouts_and_ragged_edges(cuda, la, lb, m, n, k):
    g = torch.Generator().manual_seed(m + n + k)
    A, B = _operand(m, k, la, g, cuda), _operand(k, n, lb, g, cuda)
    C = torch.full((m, n + 5), 7.0, device=cuda)
    _gemm(C, A, B, m, n, k)
    bound = 8 * 2.0**-24 * (A.abs().double() @ B.abs().double())
    assert bool(((C[:, :n].double() - A.double() @ B.double()).abs() <= bound).all())
    assert bool((C[:, n:] == 7.0).all()), "columns behind the result are written"


@pytest.mark.parametrize("n", [640, 643])
def test_accumulate(cuda, n):
    g = torch.Generator().manual_seed(n)
    A, B, C0 = (torch.randn(s, generator=g).to(cuda) for s in ((700, 512), (512, n), (700, n)))
    C = C0.clone()
    _gemm(C, A, B, 700, n, 512, accumulate=1)
    bound = 8 * 2.0**-24 * (A.abs().double() @ B.abs().double() + C0.abs().double())
    assert bool(((C.double() - (C0.double() + A.double() @ B.double())).abs() <= bound).all())


def test_values_without_a_finite_split(cuda):
    # infinities, NaN and values that round to infinity in bf16 give what fp32 arithmetic gives (tiny ones: test_gpu_gemm_f32_tiled.py)
    g = torch.Generator().manual_seed(5)
    A, B = torch.randn((600, 512), generator=g), torch.randn((512, 640), generator=g)
    B[7] *= 0.01          # (3.4e38 times it stays in range)
    A[3, 5], A[150, 7], A[599, 511], B[9, 100], B[10, 639] = float("inf"), 3.4e38, 1e-39, float("nan"), -float("inf")
    A, B = A.to(cuda), B.to(cuda)
    C = torch.zeros((600, 640), device=cuda)
    _gemm(C, A, B, 600, 640, 512)
    ref = A.double() @ B.double()
    small = ref.abs() < 1e30
    assert torch.equal(torch.isnan(C), torch.isnan(ref))
    assert bool((C[ref == float("inf")] == float("inf")).all()) and bool((C[ref == -float("inf")] == -float("inf")).all())
    bound = 512 * 2.0**-24 * (A.abs().double() @ B.abs().double())       # tiles of such values: 512 plain additions
    assert bool(((C.double() - ref).abs() <= bound)[small].all())


def test_scales_far_apart(cuda):
    # a row of tiny and a row of huge values beside ordinary ones: the split keeps each value's own 24 bits
    g = torch.Generator().manual_seed(6)
    A, B = torch.randn((600, 512), generator=g), torch.randn((512, 640), generator=g)
    A[1] *= 1e-18
    A[2] *= 1e18
    A, B = A.to(cuda), B.to(cuda)
    C = torch.zeros((600, 640), device=cuda)
    _gemm(C, A, B, 600, 640, 512)
    bound = 8 * 2.0**-24 * (A.abs().double() @ B.abs().double())
    assert bool(((C.double() - A.double() @ B.double()).abs() <= bound).all())
