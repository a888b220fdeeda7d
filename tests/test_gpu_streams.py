"""GPU: operator calls on streams of the caller's own -- several at a time, and captured into a graph.  Every result has to
have the bits of the same call made alone on the default stream: calls share weights, but no scratch and no state."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _trunk(ops, oracle, n, blocks, single_in_last=True):
    st = oracle.make_pairformer_stack_state(40 + n, blocks)
    w = ops.PackedPairformerStack(ops.PackedPairformerBlock(st, f"trunk_pairformer.{i}.", "cuda", single_in_last or i + 1 < blocks)
                                  for i in range(blocks))

    def make(seed):
        z, s, pm, sm = (t.cuda() for t in oracle.make_inputs(seed, n, pad_frac=0.1))
        return z.to(BF).contiguous(), s.to(BF).contiguous(), pm, sm

    return make, lambda z, s, pm, sm: ops.pairformer_stack_(z, s, pm, sm, w)


def _diffusion(ops, oracle, n, blocks):
    from distributed_xfold_b200 import diffusion
    st = oracle.make_diffusion_transformer_state(torch.Generator().manual_seed(n), "", 768, 384, 128, 16, blocks, 4)
    model = diffusion.PackedDiffusionTransformer(st, "", "cuda", 16, blocks, 4)
    logits = model.pair_logits(torch.randn(n, n, 128, generator=torch.Generator().manual_seed(1)).to(BF).cuda())

    def make(seed):
        g = torch.Generator().manual_seed(seed)
        act, cond = torch.randn(2, n, 768, generator=g).to(BF).cuda(), torch.randn(n, 384, generator=g).to(BF).cuda()
        return act, (torch.rand(n, generator=g) > 0.1).float().cuda(), cond

    return make, lambda act, mask, cond: (model.forward(act, mask, cond, logits),)


def _alone(make, call, seed):
    out = [t.clone() for t in call(*make(seed))]
    torch.cuda.synchronize()
    return out


CALLS = [(_trunk, dict(n=72, blocks=3)), (_trunk, dict(n=72, blocks=2, single_in_last=False)), (_diffusion, dict(n=90, blocks=4))]


@pytest.mark.parametrize("path,size", CALLS)
def test_calls_on_several_streams(ops, oracle, path, size):
    make, call = path(ops, oracle, **size)
    want = [_alone(make, call, seed) for seed in range(3)]
    streams = [torch.cuda.Stream() for _ in range(3)]
    inputs = [make(seed) for seed in range(3)]
    torch.cuda.synchronize()
    got = [[] for _ in streams]
    for _ in range(4):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                got[i].append(call(*(t.clone() for t in inputs[i])))
    ops.synchronize_and_check()
    torch.cuda.synchronize()
    for i in range(3):
        for out in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(out, want[i]))


@pytest.mark.parametrize("own_stream", [True, False])
@pytest.mark.parametrize("paths", [(0, 0, 2), (1, 2, 2)])
def test_calls_of_several_threads(ops, oracle, paths, own_stream):
    """Threads with a stream each, or all on one stream (whose scratch they share)."""
    import threading
    calls = [CALLS[i][0](ops, oracle, **CALLS[i][1]) for i in paths]
    want = [_alone(make, call, seed) for seed, (make, call) in enumerate(calls)]
    inputs = [make(seed) for seed, (make, _) in enumerate(calls)]
    torch.cuda.synchronize()
    got, gate = [[] for _ in calls], threading.Barrier(len(calls))

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.default_stream()):
            gate.wait()
            for _ in range(20):
                got[i].append(calls[i][1](*(t.clone() for t in inputs[i])))
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    ops.synchronize_and_check()
    for i in range(len(calls)):
        assert len(got[i]) == 20
        for out in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(out, want[i]))


def test_scratch_is_bounded_and_given_back(ops):
    ops._Workspace.release()
    streams = [torch.cuda.Stream() for _ in range(ops._Workspace.KEEP + 3)]
    x = torch.randn(64, 384).to(BF).cuda()
    assert len({s.cuda_stream for s in streams}) == len(streams)
    for s in streams:
        with torch.cuda.stream(s):
            first = ops._Workspace.get(x.device.index, 1000)
            assert ops._Workspace.get(x.device.index, 500) is first and ops._Workspace.get(x.device.index, 2000).numel() == 2000
    assert len(ops._Workspace._bufs) == ops._Workspace.KEEP
    ops._Workspace.release()
    assert not ops._Workspace._bufs


@pytest.mark.parametrize("path,size", CALLS)
def test_captured_call(ops, oracle, path, size):
    """A graph's scratch is its own: neither a larger call afterwards nor the release of the kept buffers touches it."""
    make, call = path(ops, oracle, **size)
    static, want = make(0), [_alone(make, call, seed) for seed in range(2)]
    st = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=st):
        out = call(*static)
    ops._Workspace.release()
    filler = torch.full((1 << 28,), 0x7F, dtype=torch.uint8, device="cuda")   # takes what has been given back
    for seed in (1, 0):
        for dst, src in zip(static, make(seed)):
            dst.copy_(src)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, want[seed]))
    ops.synchronize_and_check()
    del filler
