"""The native host path of short calls: what it takes gives the general path's results, bit by bit, in the same form;
everything else is left to the general path, whose answer (a result, a gradient, an error) stays what it was."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    assert m._host is not None, "the host path was not built"
    m.reset_device_status()  # (the status word and, below, a workspace exist from a program's first call on)
    m._decode_workspace(torch.device("cuda", torch.cuda.current_device()), m._DECODE_WS_MIN)
    return m


@pytest.fixture()
def general(ext, monkeypatch):
    """Runs a call on the general path alone."""
    def run(call):
        with monkeypatch.context() as mp:
            mp.setattr(ext, "forward_plain", ext._general)
            mp.setattr(ext, "decode_plain", ext._general)
            return call()
    return run


def _randn(*shape):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(sum(shape)), device="cuda", dtype=torch.float16)


def _same(a, b):
    assert torch.equal(a, b) and a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype
    assert a.requires_grad == b.requires_grad and a.is_inference() == b.is_inference() and a.grad_fn is b.grad_fn is None
    assert a.untyped_storage().nbytes() == b.untyped_storage().nbytes()


def _qkv(b=2, h=4, hk=2, n=65, d=64, form="bhnd"):
    if form == "bnhd":
        return [_randn(b, n, x, d).transpose(1, 2) for x in (h, hk, hk)]
    if form == "sliced":  # one projection's memory
        qkv = _randn(b, n, h + 2 * hk, d).transpose(1, 2)
        return [qkv[:, :h], qkv[:, h:h + hk], qkv[:, h + hk:]]
    return [_randn(b, x, n, d) for x in (h, hk, hk)]


FORWARD = [dict(), dict(d=32), dict(d=96, n=1), dict(d=256, n=130), dict(b=1, h=1, hk=1, n=300), dict(form="bnhd"),
           dict(form="sliced", d=128)]


@pytest.mark.parametrize("case", FORWARD)
@pytest.mark.parametrize("context", ["no_grad", "plain", "inference"])
def test_forward_is_the_general_one(ext, general, case, context):
    from flash_attn_legacy import flash_attention
    with {"no_grad": torch.no_grad, "plain": torch.enable_grad, "inference": torch.inference_mode}[context]():
        a = _qkv(**case)
        for scale in (None, 0.3):
            for causal in (False, True):
                for layout in ("bhnd", "bnhd"):
                    native = ext.forward_plain(*a, scale, causal, layout)
                    assert native is not None
                    _same(native, general(lambda: flash_attention(*a, scale, causal, layout)))


def test_forward_leaves_the_rest(ext, general):
    from flash_attn_legacy import flash_attention

    class Sub(torch.Tensor):
        pass

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    q, k, v = _qkv()
    left = lambda *a: ext.forward_plain(*a) is None  # noqa: E731
    rest = (None, False, "bhnd")
    assert not left(q, k, v, *rest)
    for bad in (q.cpu(), q.float(), q[0], q[..., ::2], q.expand(2, 4, 65, 64)[:1].expand(2, 4, 65, 64), q.as_subclass(Sub),
                _randn(2, 4, 65, 68)[..., :64], _randn(2, 4, 66, 64).flatten()[4:4 + q.numel()].view(2, 4, 65, 64),
                _randn(2, 3, 65, 64), _randn(2, 4, 64, 64), _randn(2, 4, 65, 48), None, 1.0):
        assert left(bad, k, v, *rest)
    assert left(q, v.expand(2, 2, 65, 64).requires_grad_(), v, *rest)
    assert left(q, k, v, 1, False, "bhnd") and left(q, k, v, None, 1, "bhnd") and left(q, k, v, None, False, "bshd")
    assert left(q, k, v, -1.0, False, "bhnd") and left(q, k, v, None, False) and left()
    assert left(q, _randn(2, 2, 64, 64), v, *rest) and left(q, k, _randn(2, 1, 65, 64), *rest)
    with Mode():
        assert left(q, k, v, *rest)
    with torch.overrides.BaseTorchFunctionMode():
        assert left(q, k, v, *rest)
    seen = []
    torch.func.vmap(lambda x: seen.append(left(q, x, v, *rest)) or x)(torch.stack([k, k]))
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda x: flash_attention(x, k, v))(torch.stack([q, q]))
    torch.jit.trace(lambda x: seen.append(left(x, k, v, *rest)) or x + 1, (q,), check_trace=False)
    with torch.autograd.forward_ad.dual_level():
        seen.append(left(torch.autograd.forward_ad.make_dual(q, torch.ones_like(q)), k, v, *rest))
    assert seen and all(seen)
    # gradients as before; without gradient mode the same tensors take the native path
    qg = q.detach().requires_grad_()
    assert flash_attention(qg, k, v).grad_fn is not None
    with torch.no_grad():
        assert not left(qg, k, v, *rest)
    # what is refused stays refused, what is copied stays copied
    for bad in ((q.float(), k, v), (q[..., :48].contiguous(), k, v)):
        with pytest.raises(AssertionError):
            flash_attention(*bad)
    with pytest.raises(RuntimeError):
        flash_attention(q, k, v, -1.0)
    _same(flash_attention(q, k.expand(2, 2, 65, 64), v), general(lambda: flash_attention(q, k, v)))
    assert ext.device_status() == 0


@pytest.mark.parametrize("layout", ["bshd", "bhsd"])
@pytest.mark.parametrize("b,h,hk,d,cap", [(1, 32, 8, 128, 700), (3, 4, 4, 64, 130), (2, 8, 1, 96, 300), (2, 2, 2, 256, 64)])
def test_decode_is_the_general_one(ext, general, layout, b, h, hk, d, cap):
    from flash_attn_legacy import flash_attn_with_kvcache
    caches = [_randn(b, cap, hk, d) if layout == "bshd" else _randn(b, hk, cap, d) for _ in range(2)]
    q, k, v = _randn(b, 1, h, d), _randn(b, 1, hk, d), _randn(b, 1, hk, d)
    lens = torch.randint(0, cap, (b,), dtype=torch.int32, device="cuda")
    for new in ((None, None), (k, v)):
        results = []
        for run in (lambda call: call(), general):
            kc, vc = (c.clone() for c in caches)
            out = run(lambda: flash_attn_with_kvcache(q, kc, vc, *new, cache_seqlens=lens, cache_layout=layout))
            results.append((out, kc, vc))
        for x, y in zip(*results):
            assert torch.equal(x, y) and x.stride() == y.stride()
        assert ext.decode_plain(q, *caches, *new, lens, None, layout) is not None
    # a slice of a larger cache, another stream (which gets a workspace of its own at its first call)
    kc, vc = (c[:, 1:] if layout == "bshd" else c[:, :, 1:] for c in caches)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        stream.wait_stream(torch.cuda.default_stream())
        first = flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens.clamp(max=cap - 2), cache_layout=layout)
        again = flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens.clamp(max=cap - 2), cache_layout=layout)
    stream.synchronize()
    assert torch.equal(first, again) and ext.device_status() == 0


def test_decode_leaves_the_rest(ext, general):
    from flash_attn_legacy import flash_attn_with_kvcache
    q, kc, vc, k = _randn(2, 1, 4, 64), _randn(2, 100, 2, 64), _randn(2, 100, 2, 64), _randn(2, 1, 2, 64)
    lens = torch.tensor([5, 60], dtype=torch.int32, device="cuda")
    left = lambda *a: ext.decode_plain(*a) is None  # noqa: E731
    assert not left(q, kc, vc, k, k, lens, None, "bshd")
    assert left(q, kc, vc, k, None, lens, None, "bshd") and left(q, kc, vc, None, None, None, None, "bshd")
    assert left(q, kc, vc, None, None, lens.long(), None, "bshd") and left(q, kc, vc, None, None, lens[:1], None, "bshd")
    assert left(q, kc, vc, None, None, lens, None, "bhsd") and left(q, kc, vc, None, None, lens, None, "bsdh")
    assert left(_randn(2, 2, 4, 64), kc, vc, None, None, lens, None, "bshd")
    assert left(_randn(2, 1, 8, 64)[:, :, ::2], kc, vc, None, None, lens, None, "bshd")
    assert left(q, kc, vc[:, :50], None, None, lens, None, "bshd") and left(q, kc.cpu(), vc, None, None, lens, None, "bshd")
    assert left(q, kc, vc, k[:, :, :1], k[:, :, :1], lens, None, "bshd")
    for alt in (lens.long(), lens.cpu().cuda()):
        _same(flash_attn_with_kvcache(q, kc, vc, cache_seqlens=alt),
              general(lambda: flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens)).clone())
    with pytest.raises(ValueError):
        flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, cache_layout="bsdh")
    with pytest.raises(RuntimeError):
        flash_attn_with_kvcache(q, kc, vc, k, None, cache_seqlens=lens)
    assert ext.device_status() == 0


def test_capture(ext):
    """Both calls inside a CUDA graph, replayed on new inputs."""
    from flash_attn_legacy import flash_attention, flash_attn_with_kvcache
    a = _qkv()
    q, kc, lens = _randn(1, 1, 4, 64), _randn(1, 100, 2, 64), torch.tensor([70], dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream), torch.no_grad():
        stream.wait_stream(torch.cuda.default_stream())
        for _ in range(2):
            flash_attention(*a), flash_attn_with_kvcache(q, kc, kc, cache_seqlens=lens)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            o, x = flash_attention(*a), flash_attn_with_kvcache(q, kc, kc, cache_seqlens=lens)
        a[0].neg_()
        q.neg_()
        graph.replay()
        assert torch.equal(o, flash_attention(*a)) and torch.equal(x, flash_attn_with_kvcache(q, kc, kc, cache_seqlens=lens))
    stream.synchronize()
    assert ext.device_status() == 0
