"""The weight-format kernels at the edges of their units: odd multiples of 64 columns, few rows, unaligned inputs, and every
kind of value that leaves the quantiser's short path."""
import numpy as np
import pytest
import torch

from helpers import ALL_FORMATS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e,m", ALL_FORMATS)
@pytest.mark.parametrize("rows,cols", [(256, 64), (256, 1088), (512, 576)])
def test_quantiser_takes_every_weight_like_the_definition(native_lib, e, m, rows, cols):
    """Bits of quantize_rtn -> pack -> prepack on weights drawn from ALL fp16 patterns (infinities and NaN only in rows of
    their own), on weights that sit exactly on midpoints, and with zero, negative, subnormal, infinite and NaN scales."""
    import fp6_llm_b200 as f
    from fp6_llm_b200.formats import magnitudes, pack_codes, quantize_rtn
    gen = torch.Generator().manual_seed(rows + cols)
    w = torch.randint(0, 0x7c00, (rows, cols), generator=gen, dtype=torch.int32)
    w = (w | (torch.randint(0, 2, (rows, cols), generator=gen, dtype=torch.int32) << 15)).to(torch.uint16).view(torch.float16)
    scale = (torch.rand(rows, generator=gen) * 2000 + 1e-3).half()
    scale[5], scale[6], scale[7] = 6e-8, 3e-5, 65504.0
    # rows of exact ties: midpoint * scale, where the product is an fp16 number
    mag = magnitudes(e, m)
    mid = torch.cat([(mag[:-1] + mag[1:]) / 2, mag])
    for r in range(16, 48):
        scale[r] = 2.0 ** (r - 36) * (1 + (r % 8) / 8)
        w[r] = (mid[torch.randint(0, len(mid), (cols,), generator=gen)] * scale[r].float()).half()
    w[60, ::7], w[60, 3::7], w[61, 5] = float("inf"), float("-inf"), float("-inf")
    scale[62], scale[63] = -0.5, float("inf")
    codes = quantize_rtn(w, scale, e, m)
    got = f.quantize_prepack_cuda(w.cuda(), scale.cuda(), e, m)
    expect = f.weight_prepacking_eXmY_cpu(e, m, pack_codes(codes, e, m).cuda())
    assert torch.equal(got, expect)
    # weights that start on a 4-byte but not on a 16-byte boundary
    store = torch.empty(rows * cols + 8, dtype=torch.float16, device="cuda")
    shifted = store[2:2 + rows * cols].view(rows, cols)
    shifted.copy_(w)
    assert torch.equal(f.quantize_prepack_cuda(shifted, scale.cuda(), e, m), expect)


@pytest.mark.parametrize("cols", [8, 64, 2056, 8192 + 64])
def test_row_scales_match_the_tensor_expression(native_lib, cols):
    from fp6_llm_b200 import FPxLinear
    gen = torch.Generator().manual_seed(cols)
    w = (torch.randn(37, cols, generator=gen) * 0.02).half()
    w[3], w[4, -1], w[5, 0], w[6] = 0.0, float("-inf"), float("nan"), 6e-8
    w[7, cols // 2] = -65504.0
    for e, m in ALL_FORMATS:
        from fp6_llm_b200.formats import magnitudes
        top = float(magnitudes(e, m)[-1])
        d = w.cuda()
        expect = (d.float().abs().amax(dim=1) / top).clamp_min(2.0 ** -24).to(torch.float16)
        got = FPxLinear.row_scales(d, e, m)
        assert np.array_equal(torch.nan_to_num(got, nan=-1.0).cpu().numpy(), torch.nan_to_num(expect, nan=-1.0).cpu().numpy())
        assert torch.equal(torch.isnan(got), torch.isnan(expect))


@pytest.mark.parametrize("e,m", ALL_FORMATS)
@pytest.mark.parametrize("rows,cols", [(64, 64), (128, 576), (192, 1088)])
def test_packer_and_dequantisers_at_unit_edges(native_lib, oracle_mod, e, m, rows, cols):
    """Columns that leave the last CTA, warp and lane group partly empty; every result bit-exact against the oracle."""
    import ctypes
    import fp6_llm_b200 as f
    from helpers import random_unpacked
    rng = np.random.default_rng(rows + cols + 8 * e + m)
    w = random_unpacked(rng, rows, cols, e, m)
    s = (rng.random(rows) * 0.01 + 1e-3).astype(np.float16)
    s[0], s[1], s[2] = 6e-8, 65504.0, np.inf
    d, sd = torch.from_numpy(w).cuda(), torch.from_numpy(s).cuda()
    packed = torch.empty_like(d)
    assert native_lib.fp6b200_prepack(e, m, None, d.data_ptr(), packed.data_ptr(), rows, cols) == 0   # 64-row granularity
    torch.cuda.synchronize()
    assert np.array_equal(packed.cpu().numpy(), oracle_mod.prepack(w, e, m))
    want = oracle_mod.dequant(w, s, e, m)
    same = lambda t: np.array_equal(t.cpu().numpy(), want, equal_nan=True)   # noqa: E731
    assert same(f.weight_dequant_eXmY_cpu(e, m, d, sd))
    assert same(f.dequant_packed_cuda(e, m, packed, sd))
    # a code stream that starts on an odd byte, and an fp16 result that starts on a 4-byte boundary
    raw = torch.empty(w.nbytes + 16, dtype=torch.uint8, device="cuda")
    raw[3:3 + w.nbytes] = d.view(torch.uint8).reshape(-1)
    out = torch.empty(rows, cols, dtype=torch.float16, device="cuda")
    assert native_lib.fp6b200_dequant(e, m, None, ctypes.c_void_p(raw.data_ptr() + 3), sd.data_ptr(), out.data_ptr(), rows, cols) == 0
    torch.cuda.synchronize()
    assert same(out)
    store = torch.empty(rows * cols + 8, dtype=torch.float16, device="cuda")
    assert native_lib.fp6b200_dequant_packed(e, m, None, packed.data_ptr(), sd.data_ptr(), ctypes.c_void_p(store.data_ptr() + 4), rows, cols) == 0
    torch.cuda.synchronize()
    assert same(store[2:2 + rows * cols].view(rows, cols))


def _scales_expression(w, e, m):
    from fp6_llm_b200.formats import magnitudes
    return (w.float().abs().amax(dim=1) / float(magnitudes(e, m)[-1])).clamp_min(2.0 ** -24).to(torch.float16)


def test_row_scales_stay_a_tensor_expression_where_something_watches(native_lib):
    """Gradients, vmap, forward mode, subclasses and modes see the operations; under no_grad, and inside `with torch.device`, the
    kernel gives the same values."""
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode
    from fp6_llm_b200 import FPxLinear
    gen = torch.Generator(device="cuda").manual_seed(5)
    w = torch.randn(64, 128, generator=gen, device="cuda").half()
    want = _scales_expression(w, 3, 2)
    p = torch.nn.Parameter(w)
    got = FPxLinear.row_scales(p, 3, 2)
    ref = _scales_expression(p, 3, 2)
    assert got.requires_grad and torch.equal(got, want)
    (g,), (r,) = (torch.autograd.grad(t.float().sum(), p) for t in (got, ref))
    assert torch.equal(g, r) and g.abs().sum() > 0
    with torch.no_grad():
        assert torch.equal(FPxLinear.row_scales(p, 3, 2), want)
    batched = torch.func.vmap(lambda t: FPxLinear.row_scales(t, 3, 2))(w.reshape(2, 32, 128))
    assert torch.equal(batched.reshape(-1), want)
    out, tangent = torch.func.jvp(lambda t: FPxLinear.row_scales(t, 3, 2), (w,), (torch.ones_like(w),))
    ref, ref_tangent = torch.func.jvp(lambda t: _scales_expression(t, 3, 2), (w,), (torch.ones_like(w),))
    assert torch.equal(out, want) and torch.equal(tangent, ref_tangent)

    class Counts(TorchDispatchMode):
        seen = 0

        def __torch_dispatch__(self, fn, types, args=(), kwargs=None):
            Counts.seen += fn is torch.ops.aten.amax.default
            return fn(*args, **(kwargs or {}))

    class Calls(TorchFunctionMode):
        def __torch_function__(self, fn, types, args=(), kwargs=None):
            Counts.seen += fn is torch.Tensor.amax
            return fn(*args, **(kwargs or {}))

    for mode in (Counts, Calls):
        Counts.seen = 0
        with mode():
            assert torch.equal(FPxLinear.row_scales(w, 3, 2), want)
        assert Counts.seen == 1
    with torch.device("cuda"):
        assert torch.equal(FPxLinear.row_scales(w, 3, 2), want)
    assert torch.equal(FPxLinear.row_scales(torch._neg_view(w), 3, 2), want)
