"""The fp32 GEMM's kernels through cavs_gemm_f32_tiled, each given outright: both tile widths of the tensor-core kernel, k cut over
CTAs, accumulation, every way of reading an operand, values whose three bf16 parts do not hold them, waits that run out.

Tolerance, per value and against a 64-bit product: 2^-24 of sum |a||b| for each operation that rounds on the way -- the split
of the operands and the products kept (8), two for every 64 values of k (the accumulator's additions truncate, its value is
added rounded), one per k split.  A tile of plain fp32 loops: one per value of k."""
import ctypes

import pytest
import torch

from cavs_b200 import check, lib

pytestmark = pytest.mark.gpu
ll = ctypes.c_longlong


def _p(t):
    return ctypes.c_void_p(t.data_ptr() if t is not None else 0)


def _gemm(A, B, tile_n, splits=1, C0=None, withhold=0):
    m, k = A.shape
    n = B.shape[1]
    C = torch.full((m, n + 5), 7.0, device=A.device)
    if C0 is not None:
        C[:, :n] = C0
    scratch = torch.empty(splits * m * n, device=A.device) if splits > 1 else None
    check(lib().cavs_gemm_f32_tiled(_p(C), ll(C.stride(0)), int(C0 is not None), _p(A), ll(A.stride(0)), ll(A.stride(1)), _p(B), ll(B.stride(0)),
                                    ll(B.stride(1)), m, n, k, tile_n, splits, withhold, _p(scratch),
                                    ctypes.c_size_t(4 * scratch.numel() if splits > 1 else 0),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    assert bool((C[:, n:] == 7.0).all()), "columns behind the result are written"
    return C[:, :n]


def _bound(A, B, rounds, C0=None):
    s = A.abs().double() @ B.abs().double()
    return rounds * 2.0**-24 * (s if C0 is None else s + C0.abs().double())


def _rounds(k, splits):
    return 8 + 2 * ((k + 63) // 64) + splits


def _operand(rows, cols, layout, gen, cuda):
    """layout: "row" contiguous, "pad" with an odd pitch, "col" transposed, "colpad" transposed with an odd pitch."""
    shape = (rows, cols) if layout in ("row", "pad") else (cols, rows)
    t = torch.randn((shape[0], shape[1] + (3 if layout.endswith("pad") else 0)), generator=gen).to(cuda)[:, :shape[1]]
    return t if layout in ("row", "pad") else t.t()


@pytest.mark.parametrize("tile_n", [64, 128])
@pytest.mark.parametrize("splits", [1, 2, 5, 32])
@pytest.mark.parametrize("k", [40, 512, 513, 1100])      # below a block; the corrections' drain at 8 blocks, past it, twice
def test_k_blocks_splits_and_accumulation(cuda, tile_n, splits, k):
    g = torch.Generator().manual_seed(k + splits)
    A, B, C0 = (torch.randn(s, generator=g).to(cuda) for s in ((260, k), (k, 201), (260, 201)))
    R = A.double() @ B.double()
    assert bool(((_gemm(A, B, tile_n, splits).double() - R).abs() <= _bound(A, B, _rounds(k, splits))).all())
    C = _gemm(A, B, tile_n, splits, C0)
    assert bool(((C.double() - (R + C0.double())).abs() <= _bound(A, B, _rounds(k, splits) + 1, C0)).all())


@pytest.mark.parametrize("tile_n", [64, 128])
@pytest.mark.parametrize("la", ["row", "pad", "col", "colpad"])
@pytest.mark.parametrize("lb", ["row", "pad", "col", "colpad"])
@pytest.mark.parametrize("m,n,k", [(131, 77, 150), (256, 192, 128), (388, 132, 68)])
def test_operand_layouts(cuda, tile_n, la, lb, m, n, k):
    g = torch.Generator().manual_seed(m + n + k)
    A, B = _operand(m, k, la, g, cuda), _operand(k, n, lb, g, cuda)
    assert bool(((_gemm(A, B, tile_n).double() - A.double() @ B.double()).abs() <= _bound(A, B, _rounds(k, 1))).all())


@pytest.mark.parametrize("values", ["normal", "uniform", "half-normal", "sigmoid"])
@pytest.mark.parametrize("k", [16, 64, 512, 2048])
def test_no_further_from_64_bits_than_the_cuda_cores(cuda, values, k):
    # same-signed operands with a short k are the tensor core's bad case: its additions err to one side
    g = torch.Generator().manual_seed(k)
    A, B = torch.randn((384, k), generator=g).to(cuda), torch.randn((k, 512), generator=g).to(cuda)
    if values == "uniform":
        A, B = torch.rand((384, k), generator=g).to(cuda), torch.rand((k, 512), generator=g).to(cuda)
    elif values == "half-normal":
        A, B = A.abs(), B.abs()
    elif values == "sigmoid":
        A, B = torch.sigmoid(A), torch.sigmoid(B)
    R = A.double() @ B.double()
    plain, split = ((_gemm(A, B, t).double() - R).norm() / R.norm() for t in (0, 128))
    assert split <= plain


@pytest.mark.parametrize("tile_n", [64, 128])
@pytest.mark.parametrize("exponent", [-100, -109, -112, -120, -130, -140])
def test_small_values_keep_their_bits(cuda, tile_n, exponent):
    # one row whose values fall under bf16's range (the third part first, then all of them), ordinary ones around it
    g = torch.Generator().manual_seed(-exponent)
    k = 192
    A, B = torch.randn((200, k), generator=g), torch.randn((k, 136), generator=g)
    A[77] = (A[77].double() * 2.0**exponent).float()
    A[:, 5], B[5] = A[:, 5] * 2.0**-100, B[5] * 2.0**100
    A, B = A.to(cuda), B.to(cuda)
    C = _gemm(A, B, tile_n)
    # (results may lie under fp32's smallest normal value: half a unit of the smallest subnormal for each operation)
    assert bool(((C.double() - A.double() @ B.double()).abs() <= _bound(A, B, k) + k * 2.0**-150).all())


@pytest.mark.parametrize("tile_n", [64, 128])
@pytest.mark.parametrize("splits,accumulate", [(1, False), (1, True), (3, False)])
def test_marked_tiles_among_many(cuda, tile_n, splits, accumulate):
    # several tiles per CTA, some of them computed by plain fp32 loops afterwards, beside ordinary ones
    g = torch.Generator().manual_seed(tile_n + splits)
    m, n, k = 2500, 1300, 400
    A, B = torch.randn((m, k), generator=g), torch.randn((k, n), generator=g)
    A[3, 5], A[1200, 399], A[2499, 0], A[700, 100] = float("inf"), 1e-39, float("nan"), 3.4e38
    B[:, 50] = 0
    B[100] *= 0.01
    B[17, 1299] = -float("inf")
    C0 = torch.randn((m, n), generator=g).to(cuda) if accumulate else None
    A, B = A.to(cuda), B.to(cuda)
    C = _gemm(A, B, tile_n, splits, C0)
    R = A.double() @ B.double()
    if accumulate:
        R += C0.double()
    assert torch.equal(torch.isnan(C), torch.isnan(R))
    assert bool((C[R == float("inf")] == float("inf")).all()) and bool((C[R == -float("inf")] == -float("inf")).all())
    small = R.abs() < 1e30
    assert bool(((C.double() - R).abs() <= _bound(A, B, k + splits + 1, C0))[small].all())


@pytest.mark.parametrize("tile_n", [64, 128])
@pytest.mark.parametrize("splits", [1, 3])
def test_waits_that_run_out_cost_time_not_the_result(cuda, tile_n, splits):
    # no operand is ever handed over, so that every wait of the kernel expires: plain fp32 loops give the product
    g = torch.Generator().manual_seed(9)
    A, B = torch.randn((200, 200), generator=g).to(cuda), torch.randn((200, 190), generator=g).to(cuda)
    want = _gemm(A, B, tile_n, splits, withhold=1)
    assert bool(((want.double() - A.double() @ B.double()).abs() <= _bound(A, B, 200 + splits)).all())
    assert bool(((_gemm(A, B, tile_n, splits).double() - A.double() @ B.double()).abs() <= _bound(A, B, _rounds(200, splits))).all())
