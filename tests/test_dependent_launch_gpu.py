"""Kernels that start while the kernel before them ends: inputs written, lengths moved and buffers reused on the stream
right before and after every call, directly and inside captured graphs (behind kernels, copies, memsets and joined
streams), and calls that read what the call before them wrote, give what the same calls give with a synchronisation
between all of them.  Every buffer holds something else until its producer runs, and no two passes the same inputs: what is
read too early shows."""
import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    m.reset_device_status()
    yield m
    assert m.device_status() == 0


def _work(ext, d, src, slow, step, pause, side):
    """(A chain of calls over buffers that each call's producer overwrites, the copies it leaves of everything.)"""
    steps = [torch.arange(5, device="cuda", dtype=torch.int32) * (50 + i) for i in range(3)]
    q, k, v, o, o2 = (torch.zeros_like(src[0][0]) for _ in range(5))
    lse = torch.zeros(4, 4, 200, device="cuda")
    o1 = torch.zeros(4, 4, 1, d, device="cuda", dtype=torch.float16)
    dec, dec2 = (torch.zeros(4, 4, d, device="cuda", dtype=torch.float16) for _ in range(2))
    kc, vc = (torch.zeros(4, 600, 4, d, device="cuda", dtype=torch.float16) for _ in range(2))
    lens = torch.zeros(4, dtype=torch.int32, device="cuda")
    cu = torch.zeros(5, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(ext.backward_workspace_bytes(4, 4, 200, d), dtype=torch.uint8, device="cuda")
    scale = d ** -0.5
    out = []  # (tensor, whether it is the same bit by bit: the order in which dQ is added up is not fixed)

    def produce(i):
        if step == "copy":
            for a, b in zip((q, k, v), src[i]):
                a.copy_(b)
        elif step == "memset":
            for a in (q, k, v):
                a.zero_()
        elif step == "join":
            main = torch.cuda.current_stream()
            side.wait_stream(main)
            with torch.cuda.stream(side):
                slow @ slow
                for a, b in zip((q, k, v), src[i]):
                    a.copy_(b)
            main.wait_stream(side)
        else:  # a kernel that is still busy when ours is launched
            slow @ slow
            torch.mul(src[i][0], i + 1, out=q)
            torch.add(src[i][1], slow[:1, :1], out=k)
            torch.add(src[i][2], i, out=v)

    def run():
        out.clear()
        lens.zero_()
        for i in range(3):
            for a in (q, k, v, o, o2, o1, dec, dec2, kc, vc):
                a.fill_(30)
            lse.fill_(0)
            cu.zero_()
            scratch.fill_(0x47)  # (as fp32: 51 015)
            pause()
            produce(i)
            pause()
            ext.forward(q, k, v, scale, i == 1, out=o, lse=lse)
            pause()
            ext.forward(o, k, v, scale, i == 1, out=o2)
            pause()
            grads = ext.backward(src[i][0], q, k, v, o, lse, scale, i == 1, workspace=scratch)
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
            ext.forward(q[:, :, i:i + 1], k[:, :, :1], v[:, :, :1], scale, out=o1)
            pause()
            ext.decode(o1.view(4, 4, d), kc, vc, lens, scale, o1.view(4, 4, d), o1.view(4, 4, d), out=dec)
            pause()
            ext.decode(dec, kc, vc, lens, scale, dec, o1.view(4, 4, d), out=dec2)
            pause()
            lens.add_(200)
            pause()
            chunk, _ = ext.forward_kvcache(q[:, :, :40], kc.transpose(1, 2), vc.transpose(1, 2), lens, scale)
            pause()
            lens.sub_(200)
            same = (o, lse, o2, *grads[1:], po, pl, *pg[1:], o1, dec, dec2, chunk, kc, vc)
            out.extend((x.clone(), True) for x in same)
            out.extend((x.clone(), False) for x in (grads[0], pg[0]))
            pause()
    return run, out


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("step", ["kernel", "copy", "memset", "join"])
@pytest.mark.parametrize("captured", [False, True])
def test_order(ext, d, step, captured):
    gen = torch.Generator(device="cuda").manual_seed(d)
    src = torch.randn(3, 3, 4, 4, 200, d, generator=gen, device="cuda", dtype=torch.float16)
    slow = torch.randn(2048, 2048, generator=gen, device="cuda", dtype=torch.float16)
    stream, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        run, got = _work(ext, d, src, slow, step, lambda: None, side)
        if captured:
            run()  # (a first pass outside)
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                run()
            src.mul_(-0.75)
            graph.replay()
        else:
            run()
        torch.cuda.synchronize()
        run, want = _work(ext, d, src, slow, step, torch.cuda.synchronize, side)
        run()
        torch.cuda.synchronize()
    assert len(want) == len(got) == 51
    for i, ((a, exact), (b, _)) in enumerate(zip(want, got)):
        assert torch.isfinite(a).all(), i
        if exact:
            assert torch.equal(a, b), i
        else:
            assert orc.rel_max_err(b, a.cpu()) <= orc.TOL_GRAD, i
