"""The products of the floating routes at the sizes where their tiles, splits and clipped stores can go wrong."""
import pytest
import torch

import gpu_helpers as H
from i8muon_b200 import CutlassNSInt8, check_status, native, recommend_coefficients
from oracle import ns_oracle as o

pytestmark = pytest.mark.gpu
C5 = recommend_coefficients(5)


def tf32_planes(t):
    """value = hi + lo, both rounded to the nearest TF32 value (22 significant bits)."""
    def nearest(v):
        return (v.view(torch.int32) + 0xfff + ((v.view(torch.int32) >> 13) & 1) & ~0x1fff).view(torch.float32)
    hi = nearest(t)
    return hi, nearest(t - hi)


def close(got, ref, tol):
    got, ref = got.double(), ref.double()
    return bool(((got - ref).abs() <= tol * (ref.abs() + ref.abs().mean())).all())


# (batch, m, n, k): one K block; fewer K blocks than CTAs of the largest cluster; every cluster size (few tiles with a long
# K are split most); K shares of different lengths; extents on, below and above a tile; more tiles than SMs
FP32_SHAPES = [(1, 16, 16, 16), (1, 128, 128, 96), (1, 128, 256, 4096), (2, 144, 272, 2064), (1, 512, 640, 1040),
               (1, 1024, 1024, 1024), (7, 112, 400, 48), (3, 896, 1024, 160)]


@pytest.mark.parametrize("b,m,n,k", FP32_SHAPES)
def test_fp32_products_over_all_splits(cuda_device, b, m, n, k):
    """Plain, transposed, symmetric, polynomial and final stores against float64.  The bound, 4e-6 of an entry plus the
    typical entry, is that of the other tests of these products: 22 operand bits, the low-by-low term left out, and one
    truncation of 2^-23 for each of the 12 instructions between two roundings into FP32."""
    tol = 4e-6
    gen = torch.Generator().manual_seed(m + n + k)
    l, h = m - 3, n - 5                                   # logical extents: the rest is stored as zeros
    a = torch.randn(b, m, k, generator=gen) * 0.3
    bt = torch.randn(b, n, k, generator=gen) * 0.3
    (a, a_lo), (bt, bt_lo) = tf32_planes(a.to(cuda_device)), tf32_planes(bt.to(cuda_device))
    av, bv = a.double() + a_lo.double(), bt.double() + bt_lo.double()

    ref = av @ bv.mT
    ref[:, l:] = 0
    ref[:, :, h:] = 0
    out, out_t, lo, lo_t = H.float_gemm(a, bt, lm=l, ln=h, want_t=True, left_lo=a_lo, right_lo=bt_lo)
    assert close(out + lo, ref, tol)
    assert torch.equal(out_t, out.mT) and torch.equal(lo_t, lo.mT)
    again, _, again_lo, _ = H.float_gemm(a, bt, lm=l, ln=h, want_t=True, left_lo=a_lo, right_lo=bt_lo)
    assert torch.equal(again, out) and torch.equal(again_lo, lo)

    gram, _, gram_lo, _ = H.float_gemm(a, a, sym=True, lm=l, ln=l, left_lo=a_lo, right_lo=a_lo)
    ref = av @ av.mT
    ref[:, l:] = 0
    ref[:, :, l:] = 0
    assert close(gram + gram_lo, ref, tol)
    assert torch.equal(gram, gram.mT) and torch.equal(gram_lo, gram_lo.mT)

    ca, cb, cc = C5[1]
    poly, _, poly_lo, _ = H.float_gemm(gram, gram, mode=1, sym=True, lm=l, ln=l, coeffs=(ca, cb, cc), left_lo=gram_lo,
                                       right_lo=gram_lo)
    gd = gram.double() + gram_lo.double()
    terms = abs(cb) * gd.abs() + abs(cc) * (gd.abs() @ gd.abs())
    ref = cb * gd + cc * (gd @ gd)
    ref.diagonal(dim1=1, dim2=2)[:, :l] += ca
    assert bool(((poly.double() + poly_lo.double() - ref).abs() <= 2 * tol * (terms + abs(ca))).all())

    want = (av @ bv.mT)[:, :l, :h]
    for out_dtype, unit in ((torch.float32, 0.0), (torch.bfloat16, 2.0 ** -8)):
        for transpose in (False, True):
            got, *_ = H.float_gemm(a, bt, final=True, transpose=transpose, out_dtype=out_dtype, lm=l, ln=h, left_lo=a_lo,
                                   right_lo=bt_lo)
            assert close(got, want.mT if transpose else want, tol + unit)
    assert H.status_ok(cuda_device) == 0


# the K blocks of these products form 8, 4, 2 and 1 segments; the batches take as many CTAs per tile, half as many and one
@pytest.mark.parametrize("rows,cols,batches", [(100, 1500, (1, 14, 20, 40, 160)), (512, 2048, (1, 2, 4, 7, 24)), (700, 1537, (1, 2, 6)),
                                               (1024, 1024, (1, 3)), (16, 40, (1, 300)), (256, 256, (1, 6, 12, 40)),
                                               (251, 256, (1, 6, 12, 40))])
@pytest.mark.parametrize("entry", ["_regular_prec", "_gram_prec"])
def test_fp32_results_do_not_depend_on_the_batch(cuda_device, rows, cols, batches, entry):
    x = torch.randn(max(batches), rows, cols, generator=torch.Generator().manual_seed(rows)).to(cuda_device)
    call = getattr(CutlassNSInt8(), entry)
    results = [call(x[:n], C5, 1e-7, True, "float32") for n in batches]
    check_status()
    for y in results[1:]:
        assert torch.equal(y[:1], results[0])
    assert all(torch.equal(y, results[-1][:len(y)]) for y in results)


# one matrix leaves the GPU half empty (units of one tile), the batches fill it (units of two)
@pytest.mark.parametrize("precision", ["float16", "bfloat16", "int8", "int8_bq", "fp8"])
@pytest.mark.parametrize("rows,cols", [(300, 700), (513, 257)])
def test_other_results_do_not_depend_on_the_batch_either(cuda_device, rows, cols, precision):
    x = torch.randn(40, rows, cols, generator=torch.Generator().manual_seed(rows)).to(cuda_device)
    engine = CutlassNSInt8()
    for gram in (False, True):
        function, compute = engine.router(rows, cols, precision, gram, 1.0)
        many = function(x, coeffs=C5, precision=compute)
        for n in (1, 6):
            assert torch.equal(function(x[:n], coeffs=C5, precision=compute), many[:n])
    check_status()


# extents one below, on and above a 16-bit tile; rows with no 16-byte vectors; one, odd and even tile columns
@pytest.mark.parametrize("precision", ["float16", "bfloat16"])
@pytest.mark.parametrize("batch,l,h", [(1, 16, 16), (2, 127, 129), (1, 128, 257), (3, 255, 385), (1, 130, 1030), (40, 192, 200)])
def test_16bit_calls_in_both_orientations(cuda_device, precision, batch, l, h):
    """The stored matrix keeps the caller's orientation: wide matrices read it across K in the update product, tall ones
    in the Gram product.  Both against the oracle at the tolerance of these routes."""
    x = torch.randn(batch, l, h, generator=torch.Generator().manual_seed(l + h)) * 0.02
    engine = CutlassNSInt8()
    for given in (x, x.mT.contiguous()):
        for dtype in (torch.float32, torch.bfloat16):
            v = given.to(dtype)
            y = engine._regular_prec(v.to(cuda_device), C5, 1e-7, True, precision)
            check_status()
            norm, _ = H.stats(v.to(cuda_device))
            ref = o.ns_float(v, C5, 1e-7, precision, norm=norm.cpu().numpy()).double()
            assert y.shape == v.shape and y.dtype == dtype
            assert bool(((y.double().cpu() - ref).norm(dim=(1, 2)) < 2e-2 * ref.norm(dim=(1, 2))).all())


# whole and clipped tiles, one, odd and even tile columns, extents that are no multiple of 16; wide and tall inputs
@pytest.mark.parametrize("shape", [(1, 16, 16), (2, 128, 384), (2, 127, 129), (3, 255, 400), (1, 400, 255), (1, 1030, 130), (2, 512, 256)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_int8_updates_that_read_x_across_k(cuda_device, shape, dtype):
    """Integer products are exact, so a whole call is the same bit for bit with plain dot products (the debug core) in the
    place of the tensor core's reading of X with its rows along K.  Both calls run the same quantisers, which the stage
    tests and the whole calls against the oracle hold."""
    x = (torch.randn(shape, generator=torch.Generator().manual_seed(sum(shape))) * 0.02).to(dtype).to(cuda_device)
    engine = CutlassNSInt8(fp16_first=False)
    got = engine._regular_i8(x, C5, 1e-7, True, "int8")
    native.call("i8m_set_debug_core", 1)
    try:
        want = engine._regular_i8(x, C5, 1e-7, True, "int8")
    finally:
        native.call("i8m_set_debug_core", 0)
    check_status()
    assert torch.equal(got, want)


@pytest.mark.parametrize("shape", [(2, 256, 384), (1, 100, 300)])
def test_int8_calls_take_any_epsilon(cuda_device, shape):
    """The norm of these inputs is far above both values, so neither takes part in the result."""
    x = torch.randn(shape, generator=torch.Generator().manual_seed(1)).to(cuda_device)
    engine = CutlassNSInt8(fp16_first=False)
    assert torch.equal(engine._regular_i8(x, C5, -1.0), engine._regular_i8(x, C5, 0.0))
    check_status()
