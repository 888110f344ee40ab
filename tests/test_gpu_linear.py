"""GPU parity of the linear layer, through the C interface and the Python operators.

Ground truth = the oracle's dequantisation followed by an fp32 matmul (the reference's own test recipe,
tests/python/kernel_test_fp6.py:48-58).  Tolerances, stated by the task: relative Frobenius error <= 2e-3 and,
for every output row, max |error| <= 1e-2 * max |truth| of that row."""
import numpy as np
import pytest
import torch

from helpers import FORMATS, kat_ones

pytestmark = pytest.mark.gpu

REL_FRO = 2e-3
ROW_MAX = 1e-2


def _case(oracle_mod, e, m, oc, ic, bs, seed, synth=False):
    from fp6_llm_b200.formats import random_codes_layer, synth_layer
    import fp6_llm_b200 as f
    if synth:
        w, s = synth_layer(oc, ic, e, m, seed)
    else:
        w, s = random_codes_layer(oc, ic, e, m, seed)
    x = torch.randn(bs, ic, generator=torch.Generator().manual_seed(seed + 1)).half()
    packed = f.weight_prepacking_eXmY_cpu(e, m, w.cuda())
    truth = oracle_mod.linear(x.numpy(), w.numpy(), s.numpy(), e, m)
    return packed, s.cuda(), x.cuda(), truth


def _check(oracle_mod, y, truth):
    import fp6_llm_b200 as f
    assert f.device_status() == 0, "a GEMM CTA timed out"
    res = oracle_mod.check_tolerance(y.float().cpu().numpy(), truth)
    assert res["rel_fro"] <= REL_FRO and res["max_row_rel"] <= ROW_MAX, res


@pytest.mark.parametrize("bs", [1, 7, 8, 9, 16, 17, 32, 33, 64, 65, 127, 128, 129, 200, 256, 300])
def test_batch_sweep_fp6(oracle_mod, bs):
    """Every N-tile bucket edge (16/32/64/128/256 and the second 256-wide tile)."""
    import fp6_llm_b200 as f
    packed, s, x, truth = _case(oracle_mod, 3, 2, 512, 512, bs, seed=bs)
    _check(oracle_mod, f.linear_forward_cuda(x, packed, s, 1), truth)


@pytest.mark.parametrize("e,m", FORMATS)
@pytest.mark.parametrize("split_k", [1, 2, 3, 7, 8, 11, 0])
def test_split_k(oracle_mod, e, m, split_k):
    """K = 512 has 8 K-blocks: every splitK a program may pass is taken, and how K is split is the library's choice for all of
    them (the split as asked is the C interface's: test_gpu_decomposition.py)."""
    import fp6_llm_b200 as f
    packed, s, x, truth = _case(oracle_mod, e, m, 256, 512, 12, seed=split_k + e)
    _check(oracle_mod, f.linear_forward_eXmY_cuda(e, m, x, packed, s, split_k), truth)


def test_config_4096_bs8(oracle_mod):
    """OC=IC=4096, BS=8, splitK=1, uniformly random codes, scales U(1e-3, 1e-2)."""
    import fp6_llm_b200 as f
    packed, s, x, truth = _case(oracle_mod, 3, 2, 4096, 4096, 8, seed=0)
    _check(oracle_mod, f.linear_forward_cuda(x, packed, s, 1), truth)
    # README argument order gives the same result
    y2 = f.linear_forward_cuda(packed, s, x, 1)
    _check(oracle_mod, y2, truth)


@pytest.mark.parametrize("oc,ic", [(1024, 4096), (768, 11008)])
@pytest.mark.parametrize("bs", [1, 32, 128])
def test_llama7b_like_fp6(oracle_mod, oc, ic, bs):
    """Row slices of the LLaMA-2-7B layer shapes (full K), quantised N(0, 0.02) weights, heuristic split-K."""
    import fp6_llm_b200 as f
    packed, s, x, truth = _case(oracle_mod, 3, 2, oc, ic, bs, seed=oc + bs, synth=True)
    _check(oracle_mod, f.linear_forward_cuda(x, packed, s, 0), truth)


@pytest.mark.parametrize("oc,ic", [(1280, 5120), (512, 13824)])
@pytest.mark.parametrize("bs,split_k", [(1, 1), (16, 2), (64, 4), (16, 8), (64, 0)])
def test_llama13b_like_fp5(oracle_mod, oc, ic, bs, split_k):
    import fp6_llm_b200 as f
    packed, s, x, truth = _case(oracle_mod, 2, 2, oc, ic, bs, seed=ic + bs, synth=True)
    _check(oracle_mod, f.linear_forward_eXmY_cuda(2, 2, x, packed, s, split_k), truth)


@pytest.mark.parametrize("bs", [512, 1024])
def test_prefill_like(oracle_mod, bs):
    import fp6_llm_b200 as f
    packed, s, x, truth = _case(oracle_mod, 3, 2, 512, 8192, bs, seed=bs, synth=True)
    _check(oracle_mod, f.linear_forward_cuda(x, packed, s, 1), truth)


@pytest.mark.parametrize("native", [False, True])
@pytest.mark.parametrize("bs", [1, 8, 20])
def test_weights_written_just_before(bs, native):
    """Weights that the previous kernel of the stream writes: the layer asks L2 for them before that kernel has finished, and
    must still see what it wrote."""
    import fp6_llm_b200 as f
    gen = torch.Generator(device="cuda").manual_seed(bs)
    oc, ic = 2048, 4096
    s = torch.full((oc,), 0.01, dtype=torch.float16, device="cuda")
    x = torch.randn(bs, ic, generator=gen, device="cuda").half()
    sources = []
    for _ in range(3):
        w = f.quantize_prepack_cuda(torch.randn(oc, ic, generator=gen, device="cuda").half() * 0.1, s)
        sources.append(f.native_repack(3, 2, w) if native else w)
    run = (lambda w: f.linear_forward_native(3, 2, x, w, s)) if native else (lambda w: f.linear_forward_cuda(x, w, s, 0))
    want = [run(w) for w in sources]
    held = torch.empty_like(sources[0])
    got = []
    for i in range(12):
        held.copy_(sources[i % 3])
        got.append(run(held))
    assert all(torch.equal(y, want[i % 3]) for i, y in enumerate(got)) and f.device_status() == 0


@pytest.mark.parametrize("bs", [33, 47, 48, 49, 65, 80, 81, 113, 129, 144, 145, 241, 257, 272, 289, 333, 481, 513, 530, 769])
@pytest.mark.parametrize("split_k", [0, 1, 3])
def test_tile_widths(oracle_mod, bs, split_k):
    """Batches are cut into equally wide token tiles of any multiple of 16 columns: the last token of a tile, the first of the
    next, and widths at both ends of every kernel's range, whatever splitK the call names."""
    import fp6_llm_b200 as f
    packed, s, x, truth = _case(oracle_mod, 2, 2, 512, 704, bs, seed=bs)
    _check(oracle_mod, f.linear_forward_eXmY_cuda(2, 2, x, packed, s, split_k), truth)


@pytest.mark.parametrize("e,m", FORMATS)
def test_known_answer_all_ones_full_size(e, m):
    """Reference tests' all-1.0 words: every output must equal IC exactly, at a full LLaMA-2-70B layer shape."""
    import fp6_llm_b200 as f
    oc, ic, bs = 8192, 8192, 16
    w = torch.from_numpy(kat_ones(e, m, oc, ic)).cuda()
    packed = f.weight_prepacking_eXmY_cpu(e, m, w)
    y = f.linear_forward_eXmY_cuda(e, m, torch.ones(bs, ic, dtype=torch.float16, device="cuda"), packed,
                                   torch.ones(oc, dtype=torch.float16, device="cuda"), 0)
    assert f.device_status() == 0
    assert torch.all(y == float(ic))


def test_full_size_against_fp16_matmul():
    """LLaMA-2-70B gate+up shape at BS=64: compare with an fp32-accumulated matmul of the GPU-dequantised weights
    (size-independent check; the dequantised weights themselves are bit-exact with the oracle, see the formats tests)."""
    import fp6_llm_b200 as f
    from fp6_llm_b200.formats import synth_layer
    oc, ic, bs = 57344, 8192, 64
    w, s = synth_layer(oc, ic, 3, 2, seed=1, device="cuda")
    packed = f.weight_prepacking_cpu(w)
    del w
    x = torch.randn(bs, ic, device="cuda", dtype=torch.float16)
    y = f.linear_forward_cuda(x, packed, s, 0)
    assert f.device_status() == 0
    w16 = f.dequant_packed_cuda(3, 2, packed, s)
    truth = (x.float() @ w16.float().T)
    rel = ((y.float() - truth).norm() / truth.norm()).item()
    row = ((y.float() - truth).abs().amax(dim=1) / truth.abs().amax(dim=1)).max().item()
    assert rel <= REL_FRO and row <= ROW_MAX, (rel, row)


def test_linearity_in_activations(oracle_mod):
    """f(x1 + x2) == f(x1) + f(x2) up to fp16 output rounding."""
    import fp6_llm_b200 as f
    packed, s, x, _ = _case(oracle_mod, 3, 2, 512, 1024, 8, seed=2)
    x1 = (x * 0.5)
    y = f.linear_forward_cuda(x, packed, s, 1).float()
    y1 = f.linear_forward_cuda(x1, packed, s, 1).float()
    assert torch.allclose(y1 * 2, y, rtol=2e-3, atol=1e-4)


def test_host_io_entry(oracle_mod):
    import fp6_llm_b200 as f
    packed, s, x, truth = _case(oracle_mod, 3, 2, 1024, 1024, 24, seed=6)
    xh = x.cpu().pin_memory()
    out = torch.empty(24, 1024, dtype=torch.float16).pin_memory()
    f.linear_forward_host(3, 2, xh, packed, s, out, 0)
    _check(oracle_mod, out, truth)


def test_error_behaviour(oracle_mod, native_lib):
    import fp6_llm_b200 as f
    packed, s, x, _ = _case(oracle_mod, 3, 2, 256, 256, 4, seed=1)
    with pytest.raises(ValueError):
        f.linear_forward_cuda(x[:, :128].contiguous(), packed, s, 1)        # K mismatch
    with pytest.raises(ValueError):
        f.linear_forward_cuda(x.float(), packed, s, 1)                      # dtype
    with pytest.raises(ValueError):
        f.linear_forward_cuda(x, packed, s[:128], 1)                        # scale length
    with pytest.raises(ValueError):
        f.linear_forward_eXmY_cuda(4, 3, x, packed, s, 1)                   # unsupported format
    out = torch.empty(4, 256, dtype=torch.float16, device="cuda")
    bad = 1   # cudaErrorInvalidValue
    assert native_lib.fp6b200_linear(3, 2, None, packed.data_ptr(), s.data_ptr(), x.data_ptr(), out.data_ptr(), 128, 4, 256, None, 1) == bad
    assert native_lib.fp6b200_linear(3, 2, None, packed.data_ptr(), s.data_ptr(), x.data_ptr(), out.data_ptr(), 256, 4, 96, None, 1) == bad
    assert native_lib.fp6b200_linear(3, 2, None, packed.data_ptr(), s.data_ptr(), x.data_ptr(), out.data_ptr(), 256, 0, 256, None, 1) == bad
    assert native_lib.fp6b200_linear(3, 2, None, packed.data_ptr(), s.data_ptr(), x.data_ptr(), out.data_ptr(), 256, 4, 256, None, 2) == bad
    assert native_lib.fp6b200_linear(1, 2, None, packed.data_ptr(), s.data_ptr(), x.data_ptr(), out.data_ptr(), 256, 4, 256, None, 1) == bad


def test_static_weights_option_gives_identical_results(native_lib):
    """With the static-weights promise the GEMM requests its weights while the previous kernel of the stream is still
    finishing; the weights here are prepacked and synchronised first, so the results must not change by a bit."""
    import fp6_llm_b200 as f
    from fp6_llm_b200.formats import random_codes_layer
    layers = []
    for i, (oc, ic) in enumerate(((4096, 4096), (1536, 2048), (512, 11008))):
        w, s = random_codes_layer(oc, ic, 3, 2, seed=20 + i, scale_lo=0.01, scale_hi=0.1)
        layers.append((f.weight_prepacking_cpu(w.cuda()), s.cuda(), torch.randn(8 + 24 * i, ic, generator=torch.Generator().manual_seed(i)).half().cuda()))
    torch.cuda.synchronize()
    assert not f.static_weights()
    plain = [f.linear_forward_cuda(x, p, s, 0) for p, s, x in layers]
    try:
        f.set_static_weights(True)
        assert f.static_weights()
        for _ in range(3):                                   # back to back on one stream: each GEMM follows a fix-up kernel
            fast = [f.linear_forward_cuda(x, p, s, 0) for p, s, x in layers]
            assert f.device_status() == 0
            for a, b in zip(plain, fast):
                assert torch.equal(a, b)
    finally:
        f.set_static_weights(False)
    assert native_lib.fp6b200_set_option(99, 1) == 1         # unknown option: cudaErrorInvalidValue
    assert native_lib.fp6b200_get_option(99) == -1


def test_module_wrapper_matches_dequantised_linear(native_lib):
    """FPxLinear.from_linear quantises and packs on the GPU; its output equals the fp32 matmul on the dequantised
    weights (plus bias) within the linear layer's tolerance, for batched inputs of any leading shape."""
    import fp6_llm_b200 as f
    torch.manual_seed(3)
    lin = torch.nn.Linear(1024, 512, bias=True).cuda().half()
    layer = f.FPxLinear.from_linear(lin)
    assert (layer.in_features, layer.out_features) == (1024, 512)
    x = torch.randn(3, 5, 1024, device="cuda").half()
    y = layer(x)
    assert y.shape == (3, 5, 512) and y.dtype == torch.float16
    w16 = f.dequant_packed_cuda(3, 2, layer.weight, layer.scales).float()
    ref = x.float().reshape(-1, 1024) @ w16.T + lin.bias.float()
    err = (y.float().reshape(-1, 512) - ref).norm() / ref.norm()
    assert err.item() <= 2e-3
    # the quantised layer stays close to the fp16 layer it came from (6-bit weights: a few percent)
    full = lin(x).float()
    assert ((y.float() - full).norm() / full.norm()).item() < 0.06
    assert f.device_status() == 0


@pytest.mark.parametrize("oc,ic,bs", [(2048, 16384, 300), (1024, 8192, 40), (1536, 12288, 130)])
def test_long_k_repeated_launches_stay_exact_per_tile(native_lib, oc, ic, bs):
    """Many pipeline stages per CTA (long K), several launches back to back: every 32-row x n-tile block of every
    launch must be within tolerance, not just the matrix as a whole (a role that misreads a ring slot's phase
    corrupts one 64-wide K block of one 32-row group, far below the whole-matrix tolerance)."""
    import fp6_llm_b200 as f
    from fp6_llm_b200.formats import random_codes_layer
    w, s = random_codes_layer(oc, ic, 3, 2, seed=oc + bs, scale_lo=0.01, scale_hi=0.1)
    packed = f.weight_prepacking_cpu(w.cuda())
    s = s.cuda()
    x = torch.randn(bs, ic, generator=torch.Generator().manual_seed(5)).half().cuda()
    ref = x.float() @ f.dequant_packed_cuda(3, 2, packed, s).float().T            # [bs, oc]
    outs = [f.linear_forward_cuda(x, packed, s, 0) for _ in range(6)]             # back to back on one stream
    assert f.device_status() == 0
    refg = ref.T.reshape(oc // 32, 32 * bs)
    for y in outs:
        err = (y.float() - ref).T.reshape(oc // 32, 32 * bs)
        rel = err.norm(dim=1) / refg.norm(dim=1)
        assert rel.max().item() <= 2e-3, (rel.argmax().item(), rel.max().item())
        assert torch.equal(y, outs[0])                                            # and the launches agree bit for bit


@pytest.mark.parametrize("oc,ic,bs", [(512, 256, 200), (1024, 2048, 300), (4096, 1024, 512)])
def test_cta_pair_tiles_give_the_same_layer(oracle_mod, native_lib, oc, ic, bs):
    """FP6B200_OPTION_PAIR_TILES: two CTAs share a 256-row tile (cta_group::2 MMAs, half of the activation tile each).
    Same tolerances against the oracle; the option is restored afterwards."""
    import fp6_llm_b200 as f
    from fp6_llm_b200.formats import random_codes_layer
    w, s = random_codes_layer(oc, ic, 3, 2, seed=oc + bs, scale_lo=0.005, scale_hi=0.02)
    x = torch.randn(bs, ic, generator=torch.Generator().manual_seed(2)).half()
    packed = f.weight_prepacking_eXmY_cpu(3, 2, w.cuda())
    truth = oracle_mod.linear(x.numpy(), w.numpy(), s.numpy(), 3, 2)
    before = native_lib.fp6b200_get_option(3)
    try:
        assert native_lib.fp6b200_set_option(3, 2) == 0
        y = f.linear_forward_eXmY_cuda(3, 2, x.cuda(), packed, s.cuda(), 0)
        assert f.device_status() == 0
    finally:
        native_lib.fp6b200_set_option(3, before)
    res = oracle_mod.check_tolerance(y.float().cpu().numpy(), truth)
    assert res["ok"], res
    plain = f.linear_forward_eXmY_cuda(3, 2, x.cuda(), packed, s.cuda(), 0)
    assert (y.float() - plain.float()).abs().max().item() <= 2e-3 * plain.float().abs().max().item()
