"""GPU parity of the DiffusionTransformer composition (AdaLN, AttentionPairBias 16 x 48, AdaLN-Zero,
DiffusionTransition) against the CPU oracle, whose forward is pinned to the reference's
DistributeDiffusionTransformer.forward.  bf16 tolerance: relative Frobenius <= 2e-2 on the activations
and <= 3e-2 on the accumulated update."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def relf(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


# the last case is the full depth of the reference's transformer (24 blocks in 6 super-blocks of 4,
# nn/d_diffusion_transformer.py:267-310) at a size the CPU oracle finishes in seconds
@pytest.mark.parametrize("n,samples,blocks", [(96, 1, 4), (150, 2, 8), (128, 1, 24)])
def test_diffusion_transformer(ops, oracle, n, samples, blocks):
    from distributed_xfold_b200 import diffusion
    g = torch.Generator().manual_seed(1000 + n)
    st = oracle.make_diffusion_transformer_state(g, "", 768, 384, 128, 16, blocks, 4)
    act = torch.randn(samples, n, 768, generator=g).to(BF)
    cond = torch.randn(n, 384, generator=g).to(BF)
    pair = torch.randn(n, n, 128, generator=g).to(BF)
    mask = (torch.rand(n, generator=g) > 0.1).float()
    rst = {k: v.to(BF).float() for k, v in st.items()}
    with torch.no_grad():
        ref = oracle.diffusion_transformer(rst, "", act.float(), mask, cond.float(), pair.float(), 16, blocks, 4)
    model = diffusion.PackedDiffusionTransformer(st, "", "cuda", 16, blocks, 4)
    pl = model.pair_logits(pair.cuda().contiguous())
    a = act.cuda().contiguous()
    model.forward(a, mask.cuda(), cond.cuda().contiguous(), pl)
    ops.synchronize_and_check()
    got = a.float().cpu()
    valid = mask > 0
    assert torch.isfinite(got).all()
    assert relf(got[:, valid], ref[:, valid]) < 2e-2
    assert relf((got - act.float())[:, valid], (ref - act.float())[:, valid]) < 3e-2


@pytest.mark.parametrize("blocks,super_block", [(3, 1), (4, 2)])
def test_diffusion_transformer_of_four_heads(ops, oracle, blocks, super_block):
    """Head counts that do not fill the sixteens in which the pair logits are computed; a narrow model."""
    from distributed_xfold_b200 import diffusion
    n, samples, c, heads = 70, 3, 128, 4
    g = torch.Generator().manual_seed(blocks)
    st = oracle.make_diffusion_transformer_state(g, "", c, 384, 128, heads, blocks, super_block)
    act, cond = torch.randn(samples, n, c, generator=g).to(BF), torch.randn(n, 384, generator=g).to(BF)
    pair, mask = torch.randn(n, n, 128, generator=g).to(BF), (torch.rand(n, generator=g) > 0.1).float()
    with torch.no_grad():
        ref = oracle.diffusion_transformer({k: v.to(BF).float() for k, v in st.items()}, "", act.float(), mask, cond.float(),
                                           pair.float(), heads, blocks, super_block)
    model = diffusion.PackedDiffusionTransformer(st, "", "cuda", heads, blocks, super_block)
    got = model.forward(act.cuda(), mask.cuda(), cond.cuda(), model.pair_logits(pair.cuda()))
    ops.synchronize_and_check()
    assert relf(got.float().cpu()[:, mask > 0], ref[:, mask > 0]) < 2e-2


def test_diffusion_single_sample_2d_input(ops, oracle):
    """[N, 768] activations (use_batch_infer False in the reference) take the same path."""
    from distributed_xfold_b200 import diffusion
    n, blocks = 64, 4
    g = torch.Generator().manual_seed(77)
    st = oracle.make_diffusion_transformer_state(g, "", 768, 384, 128, 16, blocks, 4)
    act = torch.randn(n, 768, generator=g).to(BF)
    cond = torch.randn(n, 384, generator=g).to(BF)
    pair = torch.randn(n, n, 128, generator=g).to(BF)
    mask = torch.ones(n)
    rst = {k: v.to(BF).float() for k, v in st.items()}
    with torch.no_grad():
        ref = oracle.diffusion_transformer(rst, "", act.float(), mask, cond.float(), pair.float(), 16, blocks, 4)
    model = diffusion.PackedDiffusionTransformer(st, "", "cuda", 16, blocks, 4)
    a = act.cuda().contiguous()
    model.forward(a, mask.cuda(), cond.cuda().contiguous(), model.pair_logits(pair.cuda().contiguous()))
    ops.synchronize_and_check()
    assert relf(a.float().cpu(), ref) < 2e-2


@pytest.mark.parametrize("n,samples,blocks", [(40, 1, 2), (300, 2, 24), (1900, 1, 3)])
def test_step_is_the_composition_of_its_operators(ops, oracle, n, samples, blocks):
    """The one-call step against the same blocks put together from the single operators: the same roundings at the same
    places, hence the same bits.  The conditioning of 24 blocks at 300 tokens comes in two groups, the second one shorter;
    of three blocks at 1900 tokens in groups of two and one."""
    from distributed_xfold_b200 import diffusion
    c, heads = 768, 16
    g = torch.Generator().manual_seed(n + blocks)
    st = oracle.make_diffusion_transformer_state(g, "", c, 384, 128, heads, blocks, 1)
    for k, v in st.items():
        if k.endswith("single_cond_layer_norm.weight"):
            st[k] = 1.0 + 0.3 * torch.randn(v.shape, generator=g)
    model = diffusion.PackedDiffusionTransformer(st, "", "cuda", heads, blocks, 1)
    act = torch.randn(samples, n, c, generator=g).to(BF).cuda()
    cond = torch.randn(n, 384, generator=g).to(BF).cuda()
    mask = (torch.rand(n, generator=g) > 0.1).float().cuda()
    logits = [torch.randn(1, heads, n, n, device="cuda") for _ in range(blocks)]
    prepared = [ops.prepare_pair_bias(t[0])[None] for t in logits]
    got = model.forward(act.clone(), mask, cond, prepared)
    want = act.clone()
    for i, blk in enumerate(model.blocks):
        for part, p in enumerate((f"self_attention.{i}.", f"transition_block.{i}.")):
            xn = diffusion._PackedAdaLN(st, p + "adaptive_layernorm.", "cuda")(want, cond)
            wc = st[p + "adaptive_zero_init.adaptive_zero_cond.weight"].to(BF).cuda()
            gate = ops.linear(cond, wc, st[p + "adaptive_zero_init.adaptive_zero_cond.bias"].cuda())
            if part == 0:
                o, w = ops.attention_pair_bias_core(xn, blk.att, prepared[i][0], mask), blk.att.w_out
            else:
                o, w = ops.linear_swiglu(xn, blk.tr_w1), blk.tr_w2
            ops.linear_gate_residual(o, w, gate, want, row_gate_mod=n, out=want)
    ops.synchronize_and_check()
    assert torch.isfinite(got).all() and torch.equal(got, want)


def test_pair_logits_come_in_any_list_that_covers_the_blocks(ops, oracle):
    """Per super-block a tensor or its blocks one by one, prepared or plain, more than the blocks need; too few are an error
    before anything runs, in Python and in C."""
    import ctypes
    from distributed_xfold_b200 import _cabi, diffusion
    n, blocks, sb = 40, 5, 2
    g = torch.Generator().manual_seed(8)
    st = oracle.make_diffusion_transformer_state(g, "", 768, 384, 128, 16, blocks, sb)
    model = diffusion.PackedDiffusionTransformer(st, "", "cuda", 16, blocks, sb)
    act, cond = torch.randn(n, 768, generator=g).to(BF).cuda(), torch.randn(n, 384, generator=g).to(BF).cuda()
    plain = [torch.randn(sb, 16, n, n, generator=g).cuda() for _ in range(4)]
    prepared = [ops.prepare_pair_bias(t.reshape(-1, n, n)).reshape(sb, 16, n, n) for t in plain]
    want = model.forward(act.clone(), None, cond, prepared[:3])
    for logits in (prepared, plain, [prepared[0], plain[1], prepared[2]], [list(t) for t in prepared], torch.stack(prepared),
                   prepared[:2] + [prepared[2][:1]], [torch.stack([t, t], 1)[:, 0] for t in prepared]):
        assert torch.equal(model.forward(act.clone(), None, cond, logits), want)
    with pytest.raises(IndexError):
        model.forward(act.clone(), None, cond, prepared[:2])
    lib = _cabi.load()
    ws = ops._Workspace.get(0, lib.xfold_diffusion_workspace_bytes(1, n, ctypes.byref(model.c)))
    ptrs = (ctypes.c_void_p * blocks)(*[t.data_ptr() for t in prepared])
    assert not ptrs[4]
    rc = lib.xfold_diffusion_transformer_fwd(_cabi.ctx(0), act.data_ptr(), 1, n, None, cond.data_ptr(), ctypes.byref(model.c),
                                             ptrs, ws.data_ptr(), ws.numel(), ops._stream(0))
    assert rc == _cabi.XFOLD_ERR_ARG
    ops.synchronize_and_check()


@pytest.mark.parametrize("which", ["act", "cond"])
def test_unaligned_inputs_are_refused(ops, oracle, which):
    """Activations or conditioning that start at an odd element: an error before anything runs."""
    from distributed_xfold_b200 import _cabi, diffusion
    n = 24
    g = torch.Generator().manual_seed(9)
    model = diffusion.PackedDiffusionTransformer(oracle.make_diffusion_transformer_state(g, "", 768, 384, 128, 16, 1, 1), "",
                                                 "cuda", 16, 1, 1)
    buf = torch.ones(n * 768 + 8, dtype=BF, device="cuda")
    shift = lambda width, by: buf[by:by + n * width].view(n, width)
    act, cond = shift(768, int(which == "act")), shift(384, int(which == "cond"))
    with pytest.raises(_cabi.XfoldError, match="aligned"):
        model.forward(act, None, cond, [torch.zeros(1, 16, n, n, device="cuda")])
    ops.synchronize_and_check()
    assert (buf == 1).all()


def test_sampler_loop_around_the_gpu_transformer(ops, oracle):
    """The sampler of d_alphafold3.py:316-404 (host arithmetic in diffusion_head.py) driving the DiffusionTransformer on
    the GPU, against the same loop around the CPU oracle's transformer.  The atom encoder / decoder of the reference's
    denoiser are outside this path; fixed random linear maps stand in for them (positions -> token activations ->
    position update), identical on both sides, so what is compared is the transformer inside the EDM-preconditioned
    Euler loop over a few steps, with several samples batched (use_batch_infer)."""
    from distributed_xfold_b200 import diffusion, diffusion_head as dh
    n, atoms, blocks, steps, samples = 48, 4, 4, 3, 2
    g = torch.Generator().manual_seed(31)
    st = oracle.make_diffusion_transformer_state(g, "", 768, 384, 128, 16, blocks, 4)
    rst = {k: v.to(BF).float() for k, v in st.items()}
    cond = torch.randn(n, 384, generator=g).to(BF)
    pair = torch.randn(n, n, 128, generator=g).to(BF)
    seq_mask = torch.ones(n)
    atom_mask = torch.ones(n, atoms)
    enc = (torch.randn(atoms * 3, 768, generator=g) / (atoms * 3) ** 0.5).to(BF).float()   # stand-in atom encoder
    dec = (torch.randn(768, atoms * 3, generator=g) / 768 ** 0.5).to(BF).float()           # stand-in atom decoder
    levels = 160.0 * (0.05 / 160.0) ** torch.linspace(0, 1, steps + 1)

    model = diffusion.PackedDiffusionTransformer(st, "", "cuda", 16, blocks, 4)
    pl = model.pair_logits(pair.cuda().contiguous())
    cond_d, mask_d = cond.cuda().contiguous(), seq_mask.cuda()

    def denoiser(transformer):
        def f(noisy, t_hat, step):
            act = ((noisy * dh.input_scaling(t_hat)).flatten(-2) @ enc).to(BF)             # [S, n, 768]
            out = transformer(act)
            upd = (torch.nn.functional.layer_norm(out.float(), (768,)) @ dec).reshape(noisy.shape)
            return dh.denoised_positions(noisy, upd, t_hat, atom_mask[None])
        return f

    def gpu_transformer(act):
        a = act.cuda().contiguous()
        model.forward(a, mask_d, cond_d, pl)
        ops.synchronize_and_check()
        return a.cpu()

    def cpu_transformer(act):
        with torch.no_grad():
            return oracle.diffusion_transformer(rst, "", act.float(), seq_mask, cond.float(), pair.float(), 16, blocks, 4)

    sched = dh.SamplerSchedule(levels)
    assert dh.use_batch_infer(samples, 1)
    got = dh.sample_diffusion(denoiser(gpu_transformer), sched, atom_mask, samples, generator=torch.Generator().manual_seed(5))
    ref = dh.sample_diffusion(denoiser(cpu_transformer), sched, atom_mask, samples, generator=torch.Generator().manual_seed(5))
    assert got.shape == (samples, n, atoms, 3) and torch.isfinite(got).all()
    assert relf(got, ref) < 2e-2


@pytest.mark.parametrize("n,h", [(1, 16), (77, 64), (128, 144), (130, 128), (257, 384), (50, 4), (65, 12), (130, 132)])
def test_pair_logits_prepared(ops, n, h):
    """LayerNorm + projection to the prepared pair bias at tile edges, ragged rows and head counts that fill the last
    group of heads only in part; rows with a mean well away from zero; zero in the padding columns."""
    g = torch.Generator().manual_seed(n + h)
    pair = (2.0 * torch.randn(n, n, 128, generator=g) + 0.7).to(BF)
    gamma, beta = torch.rand(128, generator=g) + 0.5, 0.3 * torch.randn(128, generator=g)
    w = torch.randn(h, 128, generator=g) / 11
    out = ops.pair_logits_prepared(pair.cuda(), gamma.cuda(), beta.cuda(), w.cuda())
    ops.synchronize_and_check()
    assert tuple(out.shape) == (h, n, (n + 7) // 8 * 8)
    ref = torch.nn.functional.layer_norm(pair.double(), (128,), gamma.double(), beta.double(), 1e-5) @ w.double().T
    ref = ref.permute(2, 0, 1) * 1.4426950408889634
    assert relf(out[..., :n].cpu(), ref) < 4e-4  # float16 output rounding only
    assert float(out[..., n:].float().abs().sum()) == 0.0


@pytest.mark.parametrize("n", [1, 40, 129, 300])
def test_pair_logits_of_few_heads_have_the_bits_of_many(ops, n):
    """Up to 96 heads go through the form with keys as the accumulator's rows, more through the one with heads as its rows:
    the same operands and sums.  Rows far from zero (mean 30, deviation 1): the mean falls out of the product with weights
    that add up to zero, whose float32 rounding leaves about 30 * 2^-24 * sqrt(128) of a weight, 2e-5; the rest is float16's
    rounding of the result, at most 2^-11 of a value and 2.1e-4 over many."""
    g = torch.Generator().manual_seed(n)
    pair = (torch.randn(n, n, 128, generator=g) + 30).to(BF)
    gamma, beta = torch.rand(128, generator=g) + 0.5, 0.3 * torch.randn(128, generator=g)
    w = torch.randn(112, 128, generator=g) / 11
    ref = torch.nn.functional.layer_norm(pair.double(), (128,), gamma.double(), beta.double(), 1e-5) @ w.double().T
    ref = ref.permute(2, 0, 1) * 1.4426950408889634
    pair, gamma, beta, w = pair.cuda(), gamma.cuda(), beta.cuda(), w.cuda()
    many = ops.pair_logits_prepared(pair, gamma, beta, w)
    assert relf(many[..., :n].cpu(), ref) < (5e-4 if n == 1 else 3e-4)
    for h in (96, 80, 48, 33, 16):
        assert torch.equal(ops.pair_logits_prepared(pair, gamma, beta, w[:h].contiguous()), many[:h])
    ops.synchronize_and_check()


@pytest.mark.parametrize("heads", [16, 112])
@pytest.mark.parametrize("which,offset", [("pair", 1), ("pair", 4), ("prepared", 1), ("prepared", 2), ("prepared", 4)])
def test_pair_logits_at_unaligned_addresses_are_refused(ops, heads, which, offset):
    """Both tensors start at multiples of 16 bytes: anything else is an error before the first launch, and nothing is written."""
    n, lib = 20, ops.load()
    pair = torch.zeros(n * n * 128 + 8, dtype=BF, device="cuda")
    out = torch.full((heads * n * 24 + 8,), 7.0, dtype=torch.float16, device="cuda")
    w = torch.ones(heads, 128, device="cuda")
    dev = pair.device.index
    p, o = pair[offset if which == "pair" else 0:], out[offset if which == "prepared" else 0:]
    rc = lib.xfold_pair_logits_prepared_fwd(ops.ctx(dev), p.data_ptr(), n, None, None, w.data_ptr(), heads, o.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream)
    with pytest.raises(RuntimeError):
        ops.check(rc, dev, "xfold_pair_logits_prepared_fwd")
    ops.synchronize_and_check()
    assert (out == 7).all()


def test_pair_logits_of_undefined_tokens(ops):
    """A token that holds NaN or infinities gets logits of -60000 (its key is left out), as from ``prepare_pair_bias``."""
    g = torch.Generator().manual_seed(3)
    pair = torch.randn(20, 20, 128, generator=g)
    pair[4, 7, 3], pair[5, 11, 60], pair[19, 19, 127] = float("nan"), float("inf"), float("-inf")
    out = ops.pair_logits_prepared(pair.to(BF).cuda(), None, None, torch.randn(32, 128, generator=g).cuda())
    want = ops.prepare_pair_bias(torch.full((1, 8, 8), float("nan"), device="cuda"))
    ops.synchronize_and_check()
    assert (want == -60000).all()
    bad = torch.zeros(20, 24, dtype=torch.bool, device="cuda")
    bad[4, 7] = bad[5, 11] = bad[19, 19] = True
    assert (out[:, bad] == -60000).all() and (out[:, ~bad].abs() < 1000).all()
