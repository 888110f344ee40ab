"""How a layer's tiles and K blocks are dealt to the SMs: whole tiles, clusters that share a tile and add their parts in shared
memory, stream-K parts behind a fix-up kernel, and the caller's own split through the C interface.  Every route against a
64-bit product of the dequantised weights: fp16 output rounding is 2^-11 / sqrt(3) = 2.8e-4 in the 2-norm, the fp32 sums add
less than 1e-5."""
import pytest
import torch

pytestmark = pytest.mark.gpu
REL = 4e-4


def _layer(oc, ic, bs, e, m):
    import fp6_llm_b200 as f
    gen = torch.Generator(device="cuda").manual_seed(oc + ic + bs)
    w = torch.randn(oc, ic, generator=gen, device="cuda").half() * 0.02
    s = f.FPxLinear.row_scales(w, e, m)
    packed = f.quantize_prepack_cuda(w, s, e, m)
    codes = f.dequant_packed_cuda(e, m, packed, torch.ones_like(s)).double() * s.double()[:, None]
    x = torch.randn(bs, ic, generator=gen, device="cuda").half()
    bias = torch.randn(oc, generator=gen, device="cuda").half()
    return packed, s, x, bias, x.double() @ codes.T


def _rel(y, truth):
    return ((y.double() - truth).norm() / truth.norm()).item()


# one tile; K too short to share; odd K shares; few tiles and a long K; a tile per SM and two over; more, with a short K
SHAPES = [(256, 64), (256, 512), (512, 1088), (1280, 5120), (4096, 704), (5120, 2112), (12288, 512), (19200, 2048), (19200, 128),
          (37888 + 512, 576)]


@pytest.mark.parametrize("oc,ic", SHAPES)
@pytest.mark.parametrize("bs", [1, 5, 16, 40, 100, 130, 300])
def test_every_decomposition(oc, ic, bs):
    import fp6_llm_b200 as f
    packed, s, x, bias, plain = _layer(oc, ic, bs, 3, 2)
    full = plain + bias.double()
    gated = torch.nn.functional.silu(full[:, 0::2]) * full[:, 1::2]
    assert _rel(f.linear_forward_cuda(x, packed, s, 0), plain) < REL
    assert _rel(f.linear_forward_ex(3, 2, x, packed, s, 0, bias), full) < REL
    assert _rel(f.linear_forward_ex(3, 2, x, packed, s, 0, bias, f.ACT_SILU_MUL), gated) < REL
    if bs <= f.NATIVE_MAX_TOKENS:
        tiles = f.native_repack(3, 2, packed)
        assert _rel(f.linear_forward_native(3, 2, x, tiles, s), plain) < REL
        assert _rel(f.linear_forward_native(3, 2, x, tiles, s, bias, f.ACT_SILU_MUL), gated) < REL
    assert f.device_status() == 0


@pytest.mark.parametrize("oc,ic,bs", [(512, 1088, 5), (4096, 704, 16), (1280, 5120, 70), (19200, 2048, 3), (768, 2048, 300)])
@pytest.mark.parametrize("split_k", [1, 2, 3, 12, 40])
def test_callers_split_stays_in_its_workspace(native_lib, oc, ic, bs, split_k):
    """split_k * M * N floats are what the caller owns, whatever decomposition runs; none for split_k = 1.  (All of these fit the
    library's own; test_callers_split_runs_as_asked has shapes that do not.)"""
    import fp6_llm_b200 as f
    packed, s, x, _, plain = _layer(oc, ic, bs, 2, 2)
    elems = split_k * oc * bs if split_k > 1 else 0
    held = torch.full((elems + 4096,), -7.0, device="cuda")
    out = torch.empty(bs, oc, dtype=torch.float16, device="cuda")
    assert native_lib.fp6b200_linear(2, 2, torch.cuda.current_stream().cuda_stream, packed.data_ptr(), s.data_ptr(), x.data_ptr(),
                                     out.data_ptr(), oc, bs, ic, held.data_ptr() if elems else None, split_k) == 0
    assert _rel(out, plain) < REL and bool((held[elems:] == -7.0).all()) and f.device_status() == 0
    assert native_lib.fp6b200_kernel_launches(oc, bs, ic, split_k) in (1, 2)


def test_scratch_is_asked_for_only_when_needed(native_lib):
    import ctypes
    import fp6_llm_b200 as f
    asked = []
    get_t = ctypes.CFUNCTYPE(ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t)
    for (oc, ic, bs), needs in {(1024, 1024, 4): False, (10240, 8192, 4): True}.items():
        packed, s, x, _, plain = _layer(oc, ic, bs, 3, 2)
        ws = torch.empty(native_lib.fp6b200_workspace_bytes(oc, bs, ic, 0), dtype=torch.uint8, device="cuda")
        out = torch.empty(bs, oc, dtype=torch.float16, device="cuda")

        def call(answer):
            del asked[:]
            get = get_t(lambda ctx, n: asked.append(n) or answer)
            return native_lib.fp6b200_linear_scratch(3, 2, torch.cuda.current_stream().cuda_stream, packed.data_ptr(), s.data_ptr(),
                                                     x.data_ptr(), out.data_ptr(), oc, bs, ic, ctypes.cast(get, ctypes.c_void_p), None,
                                                     None, 0)
        assert call(ws.data_ptr()) == 0 and len(asked) == int(needs) and all(n <= ws.numel() for n in asked)
        assert _rel(out, plain) < REL
        if needs:
            assert call(None) == 2   # cudaErrorMemoryAllocation, nothing launched
    assert f.device_status() == 0


def test_operators_take_no_more_workspace_than_the_plan_writes(native_lib):
    """Two slots of 128 rows x the tile's columns per SM, not of the kernel's widest tile."""
    import ctypes
    import fp6_llm_b200 as f
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    asked = []
    get = ctypes.CFUNCTYPE(ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t)(lambda ctx, n: asked.append(n))   # has none to give
    for oc, ic, bs, columns in ((10240, 8192, 4, 16), (10240, 8192, 70, 80), (10240, 8192, 130, 144), (10240, 8192, 200, 208),
                                (19200, 2048, 130, 144), (19200, 2048, 300, 160), (12288, 8192, 300, 160), (11008, 4096, 140, 144)):
        packed, s, x, _, plain = _layer(oc, ic, bs, 3, 2)
        out = torch.empty(bs, oc, dtype=torch.float16, device="cuda")
        del asked[:]
        rc = native_lib.fp6b200_linear_scratch(3, 2, torch.cuda.current_stream().cuda_stream, packed.data_ptr(), s.data_ptr(), x.data_ptr(),
                                               out.data_ptr(), oc, bs, ic, ctypes.cast(get, ctypes.c_void_p), None, None, 0)
        needs = native_lib.fp6b200_kernel_launches(oc, bs, ic, 0) == 2
        assert rc == (2 if needs else 0) and len(asked) == int(needs)
        assert all(0 < n <= 2 * sms * 128 * columns * 4 for n in asked)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        y = f.linear_forward_cuda(x, packed, s, 1)
        peak = torch.cuda.max_memory_allocated() - before
        assert peak <= y.numel() * 2 + sum(asked) + (2 << 20) and _rel(y, plain) < REL
    assert f.device_status() == 0


@pytest.mark.parametrize("form", ["native", "python"])
def test_operators_run_without_a_workspace_when_memory_is_full(native_lib, monkeypatch, form):
    """A caller with room for the result and no more (as with splitK = 1 and no workspace before the split became the library's
    choice): the torch allocator's limit stands in for a full GPU."""
    import fp6_llm_b200 as f
    from fp6_llm_b200 import _native
    oc, ic, bs = 10240, 8192, 130
    packed, s, x, bias, plain = _layer(oc, ic, bs, 3, 2)
    assert native_lib.fp6b200_kernel_launches(oc, bs, ic, 0) == 2   # wants a workspace
    if form == "python":
        monkeypatch.setattr(_native, "_host", type("Declining", (), {"linear": staticmethod(lambda *a: NotImplemented)}))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(bs, oc, dtype=torch.float16, device="cuda")
    total, rest = torch.cuda.get_device_properties(0).total_memory, []
    try:
        torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / total)
        with pytest.raises(torch.OutOfMemoryError):
            for _ in range(1000):                                   # what the pool still has in pieces a workspace fits into
                rest.append(torch.empty(20 << 20, dtype=torch.uint8, device="cuda"))
        del held                                                    # room for one result
        y = f.linear_forward_ex(3, 2, x, packed, s, 1, bias)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert _rel(y, plain + bias.double()) < REL and f.device_status() == 0


# The caller's own split (splits as partial sums in his workspace, a reduction behind) and waves of whole tiles: more tiles than
# SMs, a remainder that no cluster takes (two CTAs a tile do not fit, or K is too short to share), and less workspace than two
# slots per SM.  Splits of 4 + 5 and 3 + 2 + 2 K blocks, one block each, more splits than blocks; one and two token tiles.
CALLERS_SPLIT = [(28672, 576, 8, 2), (19200, 448, 5, 3), (19200, 448, 1, 12), (19200, 448, 40, 2), (19200, 448, 130, 2),
                 (9728, 448, 300, 2), (28672, 8192, 8, 2)]


@pytest.mark.parametrize("oc,ic,bs,split_k", CALLERS_SPLIT)
@pytest.mark.parametrize("e,m", [(3, 2), (2, 2)])
def test_callers_split_runs_as_asked(native_lib, oc, ic, bs, split_k, e, m):
    import fp6_llm_b200 as f
    packed, s, x, bias, plain = _layer(oc, ic, bs, e, m)
    blocks = ic // 64
    splits = min(split_k, blocks)
    elems = split_k * oc * bs
    stream = torch.cuda.current_stream().cuda_stream
    assert native_lib.fp6b200_kernel_launches(oc, bs, ic, split_k) == 2
    pre = plain + bias.double()
    for with_bias, activation, truth in ((False, f.ACT_NONE, plain), (True, f.ACT_NONE, pre),
                                         (True, f.ACT_SILU_MUL, torch.nn.functional.silu(pre[:, 0::2]) * pre[:, 1::2])):
        held = torch.full((elems + 4096,), float("nan"), device="cuda")
        out = torch.empty(bs, oc // 2 if activation else oc, dtype=torch.float16, device="cuda")
        assert native_lib.fp6b200_linear_ex(e, m, stream, packed.data_ptr(), s.data_ptr(), x.data_ptr(), out.data_ptr(), oc, bs, ic,
                                            held.data_ptr(), split_k, bias.data_ptr() if with_bias else None, activation) == 0
        assert _rel(out, truth) < REL
        # the route: every split left the whole product of its K blocks, in order, and nothing else was written
        parts = held[:splits * oc * bs].view(splits, bs, oc)
        assert not parts.isnan().any() and bool(held[splits * oc * bs:].isnan().all())
        assert _rel(parts.double().sum(0), plain) < 1e-5
        if activation == f.ACT_NONE and not with_bias and splits < blocks:
            codes = f.dequant_packed_cuda(e, m, packed, torch.ones_like(s))[:512].double() * s[:512].double()[:, None]
            k0 = 0
            for z in range(splits):
                k1 = k0 + (blocks // splits + (z < blocks % splits)) * 64
                assert _rel(parts[z, :, :512], x[:, k0:k1].double() @ codes[:, k0:k1].T) < 1e-5
                k0 = k1
    plainly = torch.empty(bs, oc, dtype=torch.float16, device="cuda")
    held = torch.empty(elems, device="cuda")
    assert native_lib.fp6b200_linear(e, m, stream, packed.data_ptr(), s.data_ptr(), x.data_ptr(), plainly.data_ptr(), oc, bs, ic,
                                     held.data_ptr(), split_k) == 0
    assert _rel(plainly, plain) < REL and f.device_status() == 0


@pytest.mark.parametrize("oc,ic,bs", [(19200, 448, 1), (19200, 448, 40), (28672, 448, 20), (9728, 448, 300), (37888, 64, 130)])
def test_waves_of_whole_tiles_without_a_workspace(native_lib, oc, ic, bs):
    """split_k = 1 with more tiles than SMs and a K too short to share: one kernel, some CTAs with a tile more than others."""
    import fp6_llm_b200 as f
    tiles = oc // 128 * ((bs + 255) // 256)
    assert tiles > torch.cuda.get_device_properties(0).multi_processor_count and ic < 512
    packed, s, x, bias, plain = _layer(oc, ic, bs, 3, 2)
    pre = plain + bias.double()
    stream = torch.cuda.current_stream().cuda_stream
    assert native_lib.fp6b200_kernel_launches(oc, bs, ic, 1) == 1
    for activation, truth in ((f.ACT_NONE, pre), (f.ACT_SILU_MUL, torch.nn.functional.silu(pre[:, 0::2]) * pre[:, 1::2])):
        out = torch.empty(bs, oc // 2 if activation else oc, dtype=torch.float16, device="cuda")
        assert native_lib.fp6b200_linear_ex(3, 2, stream, packed.data_ptr(), s.data_ptr(), x.data_ptr(), out.data_ptr(), oc, bs, ic, None, 1,
                                            bias.data_ptr(), activation) == 0
        assert _rel(out, truth) < REL
    assert f.device_status() == 0
