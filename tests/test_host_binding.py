"""The native host side of the layer call (csrc/torch_host.cpp) against the Python form of the same operators: it takes plain
contiguous CUDA tensors and nothing else, and whichever form runs, results, shapes and errors are the same."""
import threading

import pytest
import torch

import fp6_llm_b200 as f
from fp6_llm_b200 import _native


@pytest.fixture(scope="module")
def host(native_lib):
    return _native.host()


def test_declines_what_is_not_a_plain_cuda_call(host):
    x, w = torch.zeros(2, 64, dtype=torch.float16), torch.zeros(256, 12, dtype=torch.int32)
    s, tiles = torch.zeros(256, dtype=torch.float16), torch.zeros(2 * 12288, dtype=torch.uint8)
    assert host.linear(3, 2, x, w, s, 0, None, 0) is NotImplemented          # CPU tensors
    assert host.native(3, 2, x, tiles, s, None, 0) is NotImplemented
    assert host.layer(3, 2, x, w, tiles, s, 0, None, 0) is NotImplemented
    assert host.linear(3, 2, None, w, s, 0, None, 0) is NotImplemented
    assert host.linear(3.0, 2, x, w, s, 0, None, 0) is NotImplemented
    assert host.linear(3, 2, x, w, s, 2 ** 70, None, 0) is NotImplemented
    assert host.linear(3, 2, x) is NotImplemented and host.layer() is NotImplemented
    assert host.host_batch([]) is NotImplemented and host.host_batch([(3, 2, x, w, s, x, 0)]) is NotImplemented


def test_extension_belongs_to_one_torch_and_one_python(native_lib, monkeypatch):
    """After an upgrade the file of the old version is not the one that is looked for, built or loaded."""
    import os
    import sysconfig
    path = _native.host_path()
    assert os.path.exists(path) and torch.__version__ in os.path.basename(path) and path.endswith(sysconfig.get_config_var("EXT_SUFFIX"))
    assert not _native._stale(path, (_native.HOST_SOURCE,))
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    assert _native.host_path() != path and _native._stale(_native.host_path(), (_native.HOST_SOURCE,))


@pytest.mark.parametrize("content", [None, b"no library"])
def test_operators_do_without_the_extension(native_lib, monkeypatch, tmp_path, content):
    """A missing or unusable extension is a warning, once, and the Python form of every call."""
    import warnings
    path = tmp_path / "fp6_b200_host.so"
    if content is not None:
        path.write_bytes(content)
    monkeypatch.setattr(_native, "host_path", lambda: str(path))
    monkeypatch.setattr(_native, "_host", None)
    with pytest.warns(RuntimeWarning, match="no native host side"):
        stand_in = _native.host()
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert _native.host() is stand_in
    assert stand_in.linear(1) is stand_in.native() is stand_in.layer(1, 2) is stand_in.host_batch([]) is NotImplemented
    if torch.cuda.is_available():
        layer, x = _layer(), torch.randn(3, 256, device="cuda").half()
        assert layer(x).shape == (3, 512) and f.device_status() == 0


def _layer(oc=512, ic=256, e=3, m=2, bias=True, cls=None):
    gen = torch.Generator(device="cuda").manual_seed(oc + ic)
    w = torch.randn(oc, ic, generator=gen, device="cuda").half() * 0.02
    s = f.FPxLinear.row_scales(w, e, m)
    b = torch.randn(oc, generator=gen, device="cuda").half() if bias else None
    return (cls or f.FPxLinear)(f.quantize_prepack_cuda(w, s, e, m), s, b, e, m)


class _Declining:
    """Stands in for the binding so that the Python form runs."""
    linear = native = layer = host_batch = unwatched = staticmethod(lambda *a: NotImplemented)


@pytest.mark.gpu
@pytest.mark.parametrize("e,m", [(3, 2), (2, 2), (2, 3), (3, 1), (2, 1)])
@pytest.mark.parametrize("batch", [1, 8, 32, 33, 70, 150])
def test_same_as_the_python_form(host, monkeypatch, e, m, batch):
    for cls in (f.FPxLinear, f.FPxGateUpLinear):
        for with_bias in (False, True):
            layer = _layer(e=e, m=m, bias=with_bias, cls=cls)
            x = torch.randn(batch, 256, device="cuda").half()
            forms = [x, x.reshape(1, batch, 256), x[0], x.t().contiguous().t(), torch.nn.Parameter(x, requires_grad=False),
                     torch.cat([x, x], 1)[:, :256], x[::2]]
            for native in (False, True):
                if native:
                    layer.enable_native()
                got = [layer(t) for t in forms]
                calls = [lambda: f.linear_forward_ex(e, m, x, layer.weight, layer.scales, 2, layer.bias)]
                if native and batch <= f.NATIVE_MAX_TOKENS:
                    calls.append(lambda: f.linear_forward_native(e, m, x, layer.weight_native, layer.scales, layer.bias))
                got += [c() for c in calls]
                with monkeypatch.context() as mp:
                    mp.setattr(_native, "_host", _Declining)
                    want = [layer(t) for t in forms] + [c() for c in calls]
                for a, b in zip(got, want):
                    assert a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype and torch.equal(a, b)
    assert f.device_status() == 0


@pytest.mark.gpu
def test_host_batch_same_as_the_python_form(host, monkeypatch):
    layers = [_layer(512, 256, bias=False).enable_native(), _layer(1280, 1088, 2, 2, bias=False)]
    def batch(native):
        calls = []
        for i, layer in enumerate(layers * 3):
            act = torch.randn(1 + 20 * i, layer.in_features, generator=torch.Generator().manual_seed(i)).half().pin_memory()
            out = torch.empty(act.shape[0], layer.out_features, dtype=torch.float16, pin_memory=True)
            call = (layer.e_bits, layer.m_bits, act, layer.weight, layer.scales, out, 0)
            calls.append(call + (layer._buffers.get("weight_native"),) if native else call)
        return calls
    for native in (False, True):
        got, want = batch(native), batch(native)
        assert host.host_batch(list(got)) is True
        with monkeypatch.context() as mp:
            mp.setattr(_native, "_host", _Declining)
            f.linear_forward_host_batch(want)
        assert all(torch.equal(a[5], b[5]) for a, b in zip(got, want))
    good = batch(False)[0]
    for at, bad in ((2, good[2].float()), (2, good[2].cuda()), (2, good[2][:, :64]), (3, good[3][:256]), (5, good[5][:, :256]),
                    (5, good[5].cuda()), (0, 7)):
        call = good[:at] + (bad,) + good[at + 1:]
        assert host.host_batch([call]) is NotImplemented
        with pytest.raises(ValueError):
            f.linear_forward_host_batch([call])
    with pytest.raises(RuntimeError, match="host_io_batch failed"):   # no tokens: refused by the library, as before
        f.linear_forward_host_batch([good[:2] + (good[2][:0],) + good[3:5] + (good[5][:0],) + good[6:]])
    assert f.device_status() == 0


@pytest.mark.gpu
def test_same_errors(host):
    layer = _layer()
    x = torch.randn(4, 256, device="cuda").half()
    args = (3, 2, x, layer.weight, layer.scales)
    for bad in [(x.float(),), (x.cpu(),), (x[:, :128].contiguous(),), (x[:0],), (x[0],), (x.reshape(2, 2, 256),), (x.t(),)]:
        with pytest.raises(ValueError):
            f.linear_forward_eXmY_cuda(3, 2, bad[0], layer.weight, layer.scales, 1)
    with pytest.raises(ValueError):
        f.linear_forward_eXmY_cuda(*args, -1)
    with pytest.raises(ValueError):
        f.linear_forward_eXmY_cuda(4, 3, x, layer.weight, layer.scales, 1)
    with pytest.raises(ValueError):
        f.linear_forward_ex(*args, 0, layer.bias[:100])
    with pytest.raises(ValueError):
        f.linear_forward_ex(*args, 0, None, 5)
    with pytest.raises(ValueError):
        layer(x.float())
    with pytest.raises(ValueError):
        layer(x[:, :192])
    off = torch.empty(4 * 256 + 1, dtype=torch.float16, device="cuda")[1:].reshape(4, 256)   # 2-byte aligned: the library refuses
    with pytest.raises(RuntimeError, match="fp6b200_linear failed"):
        f.linear_forward_eXmY_cuda(3, 2, off, layer.weight, layer.scales, 1)
    with pytest.raises(RuntimeError):   # a batched tensor has no memory of its own
        torch.func.vmap(layer)(x.reshape(2, 2, 256))


@pytest.mark.gpu
def test_streams_threads_and_graphs(host):
    """Workspaces belong to a call: several threads on streams of their own, and replayed graphs beside eager calls, do not
    disturb one another."""
    layer = _layer(1536, 4096, bias=False).enable_native()
    xs = [torch.randn(n, 4096, device="cuda").half() for n in (1, 8, 40, 200)]
    want = [layer(x) for x in xs]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()), torch.no_grad():
            for _ in range(30):
                got = [layer(x) for x in xs]
            torch.cuda.current_stream().synchronize()
            wrong.extend(j for j, (a, b) in enumerate(zip(got, want)) if not torch.equal(a, b))

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = [layer(x) for x in xs]
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for _ in range(20):
        graph.replay()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not wrong and all(torch.equal(a, b) for a, b in zip(captured, want)) and f.device_status() == 0


def _replaced(layer, how):
    """The layer with its bias outside the buffers: as a Parameter, as a plain attribute, or as a property of a subclass."""
    bias = layer.bias
    if how == "parameter":
        layer.bias = torch.nn.Parameter(bias)
    else:
        del layer.bias
        if how == "attribute":
            object.__setattr__(layer, "bias", bias)
        else:
            layer.__class__ = type("Sub", (type(layer),), {"bias": property(lambda self: bias)})
    assert "bias" not in layer._buffers and torch.equal(layer.bias.detach(), bias)
    return layer


@pytest.mark.parametrize("cls", [f.FPxLinear, f.FPxGateUpLinear])
@pytest.mark.parametrize("how", ["parameter", "attribute", "property"])
def test_bias_outside_the_buffers_reaches_the_binding(monkeypatch, cls, how):
    """A bias that is no buffer any more must not look like no bias: what the binding is given, without a GPU."""
    seen = []

    class Recorder:
        layer = staticmethod(lambda *a: seen.append(a) or "taken")
    monkeypatch.setattr(_native, "_host", Recorder)
    layer = cls(torch.zeros(256, 12, dtype=torch.int32), torch.ones(256, dtype=torch.float16), torch.arange(256.0))
    x = torch.zeros(1, 64, dtype=torch.float16)
    assert layer(x) == "taken" and seen[-1][7] is layer.bias and seen[-1][4] is None
    tiles = torch.zeros(4, dtype=torch.uint8)
    layer.weight_native = torch.nn.Parameter(tiles, requires_grad=False)
    layer = _replaced(layer, how)
    layer(x)
    e, m, _, weight, native, scales, split, bias, _ = seen[-1]
    assert bias is not None and torch.equal(bias.detach(), torch.arange(256.0).half())
    assert weight is layer.weight and scales is layer.scales and torch.equal(native, tiles) and (e, m, split) == (3, 2, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("cls", [f.FPxLinear, f.FPxGateUpLinear])
@pytest.mark.parametrize("how", ["parameter", "attribute", "property"])
def test_bias_outside_the_buffers(cls, how):
    for native in (False, True):
        for batch in (1, 8, 40):
            layer = _layer(cls=cls)
            if native:
                layer.enable_native()
            x = torch.randn(batch, 256, device="cuda").half()
            want = layer(x)
            assert torch.equal(_replaced(layer, how)(x), want)
    assert f.device_status() == 0


@pytest.mark.gpu
def test_host_batch_refuses_buffers_it_would_read_past(host):
    """Nothing here is launched: the host checks raise before."""
    layer = _layer(512, 256, bias=False).enable_native()
    other = _layer(256, 256, bias=False).enable_native()
    act = torch.randn(8, 256).half().pin_memory()
    out = torch.empty(8, 512, dtype=torch.float16, pin_memory=True)
    good = (3, 2, act, layer.weight, layer.scales, out, 0, layer.weight_native)
    wide = torch.stack([layer.scales, layer.scales], 1)[:, 0]
    for at, bad in ((7, other.weight_native), (7, layer.weight_native[:-1]), (4, layer.scales[:500]), (4, layer.scales.float()), (4, wide),
                    (3, layer.weight.float()), (3, torch.stack([layer.weight, layer.weight], 2)[:, :, 0])):
        call = good[:at] + (bad,) + good[at + 1:]
        assert host.host_batch([call]) is NotImplemented
        with pytest.raises(ValueError):
            f.linear_forward_host_batch([call])
    f.linear_forward_host_batch([good])
    want = out.clone()
    f.linear_forward_host_batch([good[:7] + (torch.cat([layer.weight_native, other.weight_native]),)])   # longer than needed: as before
    assert torch.equal(out, want)
    many = torch.randn(64, 256).half().pin_memory()   # a batch that does not read the tiles does not mind them
    wide_out = torch.empty(64, 512, dtype=torch.float16, pin_memory=True)
    f.linear_forward_host_batch([good[:2] + (many,) + good[3:5] + (wide_out, 0, other.weight_native)])
    assert torch.equal(wide_out, layer(many.cuda()).cpu()) and f.device_status() == 0


@pytest.mark.gpu
def test_splits_the_library_refuses_stay_refused(host):
    """How K is split is the library's choice, but a splitK it would not take is an error all the same."""
    layer = _layer()
    x = torch.randn(4, 256, device="cuda").half()
    want = f.linear_forward_eXmY_cuda(3, 2, x, layer.weight, layer.scales, 1)
    for ok in (0, 3, 65535, True):
        assert torch.equal(f.linear_forward_eXmY_cuda(3, 2, x, layer.weight, layer.scales, ok), want)
    for bad in (65536, 2 ** 40):
        with pytest.raises(RuntimeError, match="fp6b200_linear failed: CUDA error 1"):
            f.linear_forward_eXmY_cuda(3, 2, x, layer.weight, layer.scales, bad)
        with pytest.raises(RuntimeError, match="fp6b200_linear failed"):
            f.FPxLinear(layer.weight, layer.scales, split_k=bad)(x)
    for bad in (1.0, 2.5):
        with pytest.raises(TypeError):
            f.linear_forward_eXmY_cuda(3, 2, x, layer.weight, layer.scales, bad)
    assert f.device_status() == 0
