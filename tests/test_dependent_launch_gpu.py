"""Kernels that start while the kernel before them ends: inputs written, lengths moved and buffers reused on the stream
right before and after every call, directly and inside captured graphs (behind kernels, copies, memsets and joined
streams), give what the same calls give with a synchronisation between all of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    m.reset_device_status()
    yield m
    assert m.device_status() == 0


def _work(ext, d, step, pause, side):
    """(A chain of calls over buffers that each call's producer overwrites, the copies it leaves of everything.)"""
    gen = torch.Generator(device="cuda").manual_seed(d)
    src = [torch.randn(4, 4, 200, d, generator=gen, device="cuda", dtype=torch.float16) for _ in range(3)]
    slow = torch.randn(2048, 2048, generator=gen, device="cuda", dtype=torch.float16)
    steps = [torch.arange(5, device="cuda", dtype=torch.int32) * (50 + i) for i in range(3)]
    q, k, v = (torch.zeros_like(x) for x in src)
    kc, vc = (torch.zeros(4, 600, 4, d, device="cuda", dtype=torch.float16) for _ in range(2))
    lens = torch.zeros(4, dtype=torch.int32, device="cuda")
    cu = torch.zeros(5, dtype=torch.int32, device="cuda")
    scale = d ** -0.5
    out = []

    def run():
        out.clear()
        lens.zero_()
        for i in range(3):
            if step == "copy":
                for a, b in zip((q, k, v), src):
                    a.copy_(b)
            elif step == "memset":
                for a in (q, k, v):
                    a.zero_()
            elif step == "join":
                main = torch.cuda.current_stream()
                side.wait_stream(main)
                with torch.cuda.stream(side):
                    slow @ slow
                    q.copy_(src[0])
                    k.copy_(src[1])
                    v.copy_(src[2])
                main.wait_stream(side)
            else:  # a kernel that is still busy when ours is launched
                slow @ slow
                torch.mul(src[0], i + 1, out=q)
                torch.add(src[1], slow[:1, :1], out=k)
                torch.add(src[2], i, out=v)
            pause()
            o, lse = ext.forward(q, k, v, scale, i == 1)
            pause()
            grads = ext.backward(src[i], q, k, v, o, lse, scale, i == 1)
            pause()
            cu.copy_(steps[i])
            pause()
            packed = [x.transpose(1, 2).reshape(800, 4, d)[:200 + 4 * i] for x in (q, k, v)]
            pause()
            po, pl = ext.forward_varlen(*packed, cu, cu, 60, 60, scale, True)
            pause()
            pg = ext.backward_varlen(po, *packed, po, pl, cu, cu, 60, 60, scale, True)
            pause()
            lens.add_(37)
            pause()
            kc.copy_(torch.cat([k, k, k], 2).transpose(1, 2))
            vc.copy_(torch.cat([v, v, v], 2).transpose(1, 2))
            pause()
            dec = ext.decode(q[:, :, i].contiguous(), kc, vc, lens, scale, k[:, :, 0].contiguous(), v[:, :, 0].contiguous())
            pause()
            lens.add_(200)
            pause()
            chunk, _ = ext.forward_kvcache(q[:, :, :40], kc.transpose(1, 2), vc.transpose(1, 2), lens, scale)
            pause()
            lens.sub_(200)
            out.extend(x.clone() for x in (o, lse, *grads[1:], po, pl, *pg[1:], dec, chunk, kc))
            pause()
    return run, out


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("step", ["kernel", "copy", "memset", "join"])
@pytest.mark.parametrize("captured", [False, True])
def test_order(ext, d, step, captured):
    # (dQ is left out: the order of its additions is not fixed)
    stream, side = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        run, want = _work(ext, d, step, torch.cuda.synchronize, side)
        run()
        run, got = _work(ext, d, step, lambda: None, side)
        torch.cuda.synchronize()
        if captured:
            run()  # (a first pass outside)
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                run()
            graph.replay()
        else:
            run()
        torch.cuda.synchronize()
    assert len(want) == len(got) == 33
    for i, (a, b) in enumerate(zip(want, got)):
        assert torch.equal(a, b), i
