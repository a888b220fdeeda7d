"""GPU parity of the module-level operators against the CPU oracle (and, through the golden file,
against the reference's own outputs), called through the C ABI.

The kernels compute in bf16 with fp32 accumulation; the oracle is evaluated in fp32 on the same
bf16-rounded inputs and weights.  Tolerance: relative Frobenius error <= 2e-2 on the updated
representation (the bound the task states for bf16), and <= 3e-2 on the residual UPDATE alone, which
is the stricter check because it removes the untouched part of z.  Where a mask pads tokens the
comparison is over the unpadded positions; padded positions only have to stay finite (their
softmax rows see nothing but -1e9 logits, whose fp32 spacing is 64, in both implementations).
"""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
TOL_Z, TOL_UPD = 2e-2, 3e-2


def relf(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def rounded(state):
    return {k: v.to(BF).float() for k, v in state.items()}


def make_pair(oracle, n, seed, pad=0.0):
    z, s, pm, sm = oracle.make_inputs(seed, n, pad_frac=pad)
    return z.to(BF), s.to(BF), pm, sm


def check_update(z0, z_gpu, z_ref, valid=None):
    z0, z_gpu, z_ref = z0.float(), z_gpu.float().cpu(), z_ref.float()
    assert torch.isfinite(z_gpu).all()
    if valid is not None:
        z0, z_gpu, z_ref = z0[valid], z_gpu[valid], z_ref[valid]
    e_z = relf(z_gpu, z_ref)
    e_u = relf(z_gpu - z0, z_ref - z0)
    assert e_z < TOL_Z and e_u < TOL_UPD, (e_z, e_u)
    return e_z, e_u


@pytest.mark.parametrize("outgoing", [True, False])
@pytest.mark.parametrize("n,maskkind", [(32, "ones"), (33, "rand"), (96, "binary"), (200, "rand"), (256, "none")])
def test_triangle_multiplication(ops, oracle, outgoing, n, maskkind):
    g = torch.Generator().manual_seed(100 + n)
    st = oracle.make_trimul_state(g, "")
    z = torch.randn(n, n, 128, generator=g).to(BF)
    mask = {"ones": torch.ones(n, n), "rand": torch.rand(n, n, generator=g), "none": None,
            "binary": (torch.rand(n, n, generator=g) > 0.2).float()}[maskkind]
    ref = z.float() + oracle.triangle_multiplication(rounded(st), "", z.float(), mask, outgoing)
    w = ops.PackedTriMul(st, "", "cuda")
    zd = z.cuda().contiguous()
    ops.triangle_multiplication_(zd, None if mask is None else mask.cuda(), w, outgoing)
    ops.synchronize_and_check()
    check_update(z, zd, ref)


@pytest.mark.parametrize("name", ["trimul/out/n24", "trimul/in/n24", "trimul/out/n40", "trimul/in/n40",
                                  "trimul/out/n33", "trimul/in/n33", "trimul_gloo2/out/n24", "trimul_gloo2/in/n24"])
def test_triangle_multiplication_golden(ops, oracle, golden, name):
    """Against the reference's own XSMMTriangleMultiplication.forward / gloo-sharded outputs."""
    meta, ref_upd = golden[name]["meta"], golden[name]["out"][0]
    n = meta["n"]
    g = torch.Generator().manual_seed(meta["seed"])
    st = oracle.make_trimul_state(g, "")
    z = torch.randn(n, n, 128, generator=g)
    # the generating script drew both random masks in turn, whichever it then used
    r1, r2 = torch.rand(n, n, generator=g), torch.rand(n, n, generator=g)
    mask = {"rand": r1, "ones": torch.ones(n, n), "binary": (r2 > 0.2).float()}[meta["mask"]]
    w = ops.PackedTriMul(st, "", "cuda")
    zd = z.to(BF).cuda().contiguous()
    ops.triangle_multiplication_(zd, mask.cuda(), w, meta["outgoing"])
    ops.synchronize_and_check()
    upd = zd.float().cpu() - z.to(BF).float()
    # the golden update is fp32 from fp32 inputs; the kernel saw bf16-rounded z and weights
    assert relf(upd, ref_upd) < 4e-2


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("n,pad", [(32, 0.0), (40, 0.2), (128, 0.0), (200, 0.1), (260, 0.1)])
def test_triangle_attention(ops, oracle, transpose, n, pad):
    g = torch.Generator().manual_seed(200 + n)
    st = oracle.make_grid_attention_state(g, "")
    z, _, pm, sm = make_pair(oracle, n, 300 + n, pad)
    ref = z.float() + oracle.grid_self_attention(rounded(st), "", z.float(), pm, z.float(), transpose)
    w = ops.PackedTriAttn(st, "", "cuda")
    zd = z.cuda().contiguous()
    ops.triangle_attention_(zd, pm.cuda(), w, transpose)
    ops.synchronize_and_check()
    check_update(z, zd, ref, pm > 0)


@pytest.mark.parametrize("rows,C", [((50, 50), 128), ((333,), 384), ((129, 130), 128)])
def test_transition(ops, oracle, rows, C):
    g = torch.Generator().manual_seed(400 + C)
    st = oracle.make_transition_state(g, "", C)
    x = torch.randn(*rows, C, generator=g).to(BF)
    ref = x.float() + oracle.transition(rounded(st), "", x.float())
    w = ops.PackedTransition(st, "", "cuda")
    xd = x.cuda().contiguous()
    ops.transition_(xd, w)
    ops.synchronize_and_check()
    check_update(x, xd, ref)


@pytest.mark.parametrize("B,S,C,H", [(1, 100, 384, 16), (2, 300, 768, 16), (1, 128, 384, 16), (1, 520, 768, 16)])
def test_attention_pair_bias_core(ops, oracle, B, S, C, H):
    g = torch.Generator().manual_seed(500 + S)
    st = oracle.make_self_attention_state(g, "", C, 0, False)
    xn = torch.randn(B, S, C, generator=g).to(BF)
    pb = torch.randn(H, S, S, generator=g)
    mask = (torch.rand(S, generator=g) > 0.15).float()
    r = rounded(st)
    d = C // H
    shp = (C, H, d)
    ref = oracle.gated_attention(xn.float(), 1e9 * (mask[None, None, None, :] - 1), pb,
                                 r["q_projection.weight"].T.reshape(shp), r["k_projection.weight"].T.reshape(shp),
                                 r["v_projection.weight"].T.reshape(shp), r["gating_query.weight"].T.reshape(shp), None,
                                 query_b=st["q_projection.bias"].reshape(H, d))
    w = ops.PackedSelfAttention(st, "", "cuda", H)
    out = ops.attention_pair_bias_core(xn.cuda().contiguous(), w, pb.cuda().contiguous(), mask.cuda())
    ops.synchronize_and_check()
    # the same call with the bias converted once beforehand gives the same bits
    out2 = ops.attention_pair_bias_core(xn.cuda().contiguous(), w, ops.prepare_pair_bias(pb.cuda().contiguous()), mask.cuda())
    ops.synchronize_and_check()
    assert torch.equal(out, out2)
    out = out.float().cpu().reshape(B, S, H, w.Dp)
    assert float(out[..., d:].abs().max()) == 0.0  # head padding stays zero
    assert relf(out[..., :d], ref) < 2e-2


@pytest.mark.parametrize("n,pad", [(64, 0.0), (100, 0.1), (192, 0.1)])
def test_pairformer_block(ops, oracle, n, pad):
    g = torch.Generator().manual_seed(600 + n)
    st = oracle.make_pairformer_block_state(g, "")
    z, s, pm, sm = make_pair(oracle, n, 700 + n, pad)
    rz, rs = oracle.pairformer_block(rounded(st), "", z.float(), pm, s.float(), sm)
    w = ops.PackedPairformerBlock(st, "", "cuda")
    zd, sd = z.cuda().contiguous(), s.cuda().contiguous()
    ops.pairformer_block_(zd, sd, pm.cuda(), sm.cuda(), w)
    ops.synchronize_and_check()
    check_update(z, zd, rz, pm > 0)
    check_update(s, sd, rs, sm > 0)


def test_pairformer_block_golden(ops, oracle, golden):
    """Against the reference's own DistributePairformerBlock.forward output."""
    meta = golden["ref/pairformer_block"]["meta"]
    ref_z, ref_s = golden["ref/pairformer_block"]["out"]
    n = meta["n"]
    g = torch.Generator().manual_seed(meta["seed"])
    st = oracle.make_pairformer_block_state(g, "")
    z = torch.randn(n, n, 128, generator=g)
    s = torch.randn(n, 384, generator=g)
    sm = (torch.rand(n, generator=g) > 0.15).float()
    pm = sm[:, None] * sm[None, :]
    w = ops.PackedPairformerBlock(st, "", "cuda")
    zd, sd = z.to(BF).cuda().contiguous(), s.to(BF).cuda().contiguous()
    ops.pairformer_block_(zd, sd, pm.cuda(), sm.cuda(), w)
    ops.synchronize_and_check()
    assert relf(zd.float().cpu()[pm > 0], ref_z[pm > 0]) < 2e-2
    assert relf(sd.float().cpu()[sm > 0], ref_s[sm > 0]) < 2e-2


def with_affine_norms(state, seed):
    """The factories initialise every LayerNorm with gamma = 1, beta = 0 (the reference's defaults); real checkpoints
    do not.  Perturb every 1-D parameter (LayerNorm scales and offsets, and the few Linear biases)."""
    g = torch.Generator().manual_seed(seed)
    out = {}
    for k, v in state.items():
        if v.ndim == 1 and k.endswith(".weight"):
            out[k] = 1.0 + 0.3 * torch.randn(v.shape, generator=g)
        elif v.ndim == 1 and k.endswith(".bias"):
            out[k] = v + 0.3 * torch.randn(v.shape, generator=g)
        else:
            out[k] = v
    return out


@pytest.mark.parametrize("n,pad", [(40, 0.0), (128, 0.1), (200, 0.1)])
def test_pairformer_block_with_affine_layernorms(ops, oracle, n, pad):
    """Every LayerNorm of the block with non-trivial scale and offset (pad / tile-tail sizes included)."""
    g = torch.Generator().manual_seed(1600 + n)
    st = with_affine_norms(oracle.make_pairformer_block_state(g, ""), 1700 + n)
    z, s, pm, sm = make_pair(oracle, n, 1800 + n, pad)
    rz, rs = oracle.pairformer_block(rounded(st), "", z.float(), pm, s.float(), sm)
    w = ops.PackedPairformerBlock(st, "", "cuda")
    zd, sd = z.cuda().contiguous(), s.cuda().contiguous()
    ops.pairformer_block_(zd, sd, pm.cuda(), sm.cuda(), w)
    ops.synchronize_and_check()
    check_update(z, zd, rz, pm > 0)
    check_update(s, sd, rs, sm > 0)


@pytest.mark.parametrize("outgoing", [True, False])
def test_triangle_multiplication_with_affine_layernorms(ops, oracle, outgoing):
    n = 128
    g = torch.Generator().manual_seed(1900)
    st = with_affine_norms(oracle.make_trimul_state(g, ""), 1901)
    z = (2.0 * torch.randn(n, n, 128, generator=g) + 0.7).to(BF)   # rows with a mean well away from zero
    mask = (torch.rand(n, n, generator=g) > 0.2).float()
    ref = z.float() + oracle.triangle_multiplication(rounded(st), "", z.float(), mask, outgoing)
    w = ops.PackedTriMul(st, "", "cuda")
    zd = z.cuda().contiguous()
    ops.triangle_multiplication_(zd, mask.cuda(), w, outgoing)
    ops.synchronize_and_check()
    check_update(z, zd, ref)


def test_transition_with_affine_layernorm(ops, oracle):
    g = torch.Generator().manual_seed(1950)
    st = with_affine_norms(oracle.make_transition_state(g, "", 128), 1951)
    x = (1.5 * torch.randn(40, 50, 128, generator=g) - 0.5).to(BF)
    ref = x.float() + oracle.transition(rounded(st), "", x.float())
    w = ops.PackedTransition(st, "", "cuda")
    xd = x.cuda().contiguous()
    ops.transition_(xd, w)
    ops.synchronize_and_check()
    check_update(x, xd, ref)


@pytest.mark.parametrize("case", ["golden", "ragged"])
def test_cross_attention(ops, oracle, golden, case):
    """Gated cross attention (the core of the atom cross-attention encoder / decoder) against the reference's spec-class
    output, and on sizes that are no multiples of anything."""
    if case == "golden":
        from test_cpu_oracle_golden import cross_attention_inputs
        qd, md, bb, ws = cross_attention_inputs(golden["spec/cross_attention"]["meta"])
        ref = golden["spec/cross_attention"]["out"][0]
    else:
        g = torch.Generator().manual_seed(77)
        B, S, K, c, H, D = 3, 19, 45, 128, 4, 32
        ws = {n: torch.randn(shape, generator=g) / 8 for n, shape in (("query_w", (c, H, D)), ("query_b", (1, H, D)),
              ("key_w", (c, H, D)), ("value_w", (c, H, D)), ("gating_w", (c, H, D)))}
        qd, md, bb = torch.randn(B, S, c, generator=g), torch.randn(B, K, c, generator=g), torch.randn(B, H, S, K, generator=g)
        rb = lambda t: t.to(BF).float()
        ref = oracle.cross_attention(rb(qd), rb(md), bb, rb(ws["query_w"]), ws["query_b"], rb(ws["key_w"]), rb(ws["value_w"]),
                                     rb(ws["gating_w"]))
    w = ops.PackedCrossAttention(ws["query_w"], ws["query_b"], ws["key_w"], ws["value_w"], ws["gating_w"], "cuda")
    out = ops.cross_attention(qd.to(BF).cuda(), md.to(BF).cuda(), bb.cuda(), w)
    ops.synchronize_and_check()
    assert relf(out.float().cpu(), ref) < 2e-2


@pytest.mark.parametrize("B,S,K,H,D", [(2, 1, 1, 1, 16), (1, 16, 128, 4, 64), (3, 33, 129, 5, 16), (2, 47, 260, 3, 32)])
def test_cross_attention_tile_edges(ops, oracle, B, S, K, H, D):
    """Sizes around the 16-query, 32-query, 4-head and 128-key steps of the kernel, with keys masked through the bias."""
    c = H * D if (H * D) % 8 == 0 else 128
    g = torch.Generator().manual_seed(B + S + K)
    ws = {n: torch.randn(shape, generator=g) / c ** 0.5 for n, shape in (("query_w", (c, H, D)), ("query_b", (1, H, D)),
          ("key_w", (c, H, D)), ("value_w", (c, H, D)), ("gating_w", (c, H, D)))}
    qd, md = torch.randn(B, S, c, generator=g), torch.randn(B, K, c, generator=g)
    keep = torch.rand(B, 1, 1, K, generator=g) > 0.2
    keep[..., 0] = True
    bb = torch.randn(B, H, S, K, generator=g) + 1e9 * (keep.float() - 1)
    rb = lambda t: t.to(BF).float()
    ref = oracle.cross_attention(rb(qd), rb(md), bb, rb(ws["query_w"]), ws["query_b"], rb(ws["key_w"]), rb(ws["value_w"]),
                                 rb(ws["gating_w"]))
    w = ops.PackedCrossAttention(ws["query_w"], ws["query_b"], ws["key_w"], ws["value_w"], ws["gating_w"], "cuda")
    out = ops.cross_attention(qd.to(BF).cuda(), md.to(BF).cuda(), bb.cuda(), w)
    ops.synchronize_and_check()
    assert relf(out.float().cpu(), ref) < 2e-2


@pytest.mark.parametrize("B,S,K", [(1, 1, 2), (2, 16, 8), (3, 17, 126), (149, 32, 128), (400, 31, 100), (592, 1, 2), (593, 1, 2),
                                   (593, 16, 22), (593, 16, 24), (593, 17, 2)])
def test_cross_attention_windows_have_the_bits_of_the_general_kernels(ops, B, S, K):
    """The one-kernel form for windows of up to 32 x 128, from one entry to several windows per CTA, against the same call
    with a bias that starts at an odd float, which the general kernels take; at the edges of the rule on many windows with few
    tokens."""
    g = torch.Generator().manual_seed(B + S + K)
    w = ops.PackedCrossAttention(*(torch.randn(128, 4, 32, generator=g) / 11 if i != 1 else torch.randn(1, 4, 32, generator=g)
                                   for i in range(5)), "cuda")
    qd, md = torch.randn(B, S, 128, generator=g).to(BF).cuda(), torch.randn(B, K, 128, generator=g).to(BF).cuda()
    keep = torch.rand(B, 1, 1, K, generator=g) > 0.2
    keep[..., 0] = True
    bias = (torch.randn(B, 4, S, K, generator=g) + 1e9 * (keep.float() - 1)).cuda()
    odd = torch.zeros(bias.numel() + 1, device="cuda")[1:].view_as(bias).copy_(bias)
    out, want = ops.cross_attention(qd, md, bias, w), ops.cross_attention(qd, md, odd, w)
    ops.synchronize_and_check()
    assert torch.isfinite(out).all() and torch.equal(out, want)


@pytest.mark.parametrize("where,shift", [("q", 0), ("q", 64), ("q", -64), ("m", 0), ("m", 32 * 128)])
def test_cross_attention_result_over_its_operands(ops, where, shift):
    """The result may lie over the queries' or the keys' tokens, at the same place or some elements further: as the call with a
    result of its own."""
    B, S, K = 400, 32, 128
    g = torch.Generator().manual_seed(5)
    w = ops.PackedCrossAttention(*(torch.randn(128, 4, 32, generator=g) / 11 if i != 1 else torch.randn(1, 4, 32, generator=g)
                                   for i in range(5)), "cuda")
    qd, md = torch.randn(B, S, 128, generator=g).to(BF).cuda(), torch.randn(B, K, 128, generator=g).to(BF).cuda()
    bias = torch.randn(B, 4, S, K, generator=g).cuda()
    want = ops.cross_attention(qd, md, bias, w)
    pad = 128
    room = torch.zeros(pad + (qd if where == "q" else md).numel() + pad, dtype=BF, device="cuda")
    held = room[pad:-pad].view(qd.shape if where == "q" else md.shape)
    held.copy_(qd if where == "q" else md)
    out = room[pad + shift:][:want.numel()].view(want.shape)
    q, m = (held, md) if where == "q" else (qd, held)
    lib, dev = ops.load(), qd.device.index
    ws = torch.empty(lib.xfold_cross_attention_workspace_bytes(B, S, K, 4, 32), dtype=torch.uint8, device="cuda")
    rc = lib.xfold_cross_attention_fwd(ops.ctx(dev), q.data_ptr(), m.data_ptr(), B, S, K, 128, 128, 4, 32, w.w_qg.data_ptr(),
                                       w.bias.data_ptr(), w.scale.data_ptr(), w.w_kv.data_ptr(), bias.data_ptr(), out.data_ptr(),
                                       ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    ops.check(rc, dev, "xfold_cross_attention_fwd")
    ops.synchronize_and_check()
    assert torch.equal(out, want)


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_cross_attention_bias_at_any_element(ops, offset):
    """A bias that is a view into a larger buffer starts at any float."""
    g = torch.Generator().manual_seed(offset)
    B, S, K, H, D, c = 3, 32, 128, 4, 32, 128
    qw, kw, vw, gw = (torch.randn(c, H, D, generator=g) / 11 for _ in range(4))
    w = ops.PackedCrossAttention(qw, torch.randn(1, H, D, generator=g), kw, vw, gw, "cuda")
    qd, md = torch.randn(B, S, c, generator=g).to(BF).cuda(), torch.randn(B, K, c, generator=g).to(BF).cuda()
    buf = torch.randn(B * H * S * K + 4, generator=g).cuda()
    bias = buf[offset:offset + B * H * S * K].view(B, H, S, K)
    assert bias.is_contiguous()
    out = ops.cross_attention(qd, md, bias, w)
    want = ops.cross_attention(qd, md, bias.clone(), w)
    ops.synchronize_and_check()
    assert torch.equal(out, want)


def test_cross_attention_result_at_any_element(ops):
    """The C entry point writes to whatever element the caller's result starts at."""
    from distributed_xfold_b200 import _cabi
    g = torch.Generator().manual_seed(5)
    B, S, K, H, D, c = 2, 19, 45, 4, 32, 128
    qw, kw, vw, gw = (torch.randn(c, H, D, generator=g) / 11 for _ in range(4))
    w = ops.PackedCrossAttention(qw, torch.randn(1, H, D, generator=g), kw, vw, gw, "cuda")
    qd, md = torch.randn(B, S, c, generator=g).to(BF).cuda(), torch.randn(B, K, c, generator=g).to(BF).cuda()
    bias = torch.randn(B, H, S, K, generator=g).cuda()
    want = ops.cross_attention(qd, md, bias, w)
    buf = torch.full((B * S * H * D + 2,), 9.0, dtype=BF, device="cuda")
    lib = _cabi.load()
    ws = ops._Workspace.get(0, lib.xfold_cross_attention_workspace_bytes(B, S, K, H, D))
    rc = lib.xfold_cross_attention_fwd(_cabi.ctx(0), qd.data_ptr(), md.data_ptr(), B, S, K, c, c, H, D, w.w_qg.data_ptr(),
                                       w.bias.data_ptr(), w.scale.data_ptr(), w.w_kv.data_ptr(), bias.data_ptr(),
                                       buf[1:].data_ptr(), ws.data_ptr(), ws.numel(), ops._stream(0))
    ops.synchronize_and_check()
    assert rc == 0 and torch.equal(buf[1:-1].view_as(want), want) and buf[0] == 9.0 and buf[-1] == 9.0


@pytest.mark.parametrize("B,S,C,H", [(4, 65, 384, 16), (3, 33, 384, 16), (1, 129, 384, 16), (2, 1100, 384, 16), (1, 64, 768, 16),
                                     (3, 400, 768, 16)])
def test_attention_reference_exponent_moves_far(ops, oracle, B, S, C, H):
    """Logits of several hundred that grow along the keys: the running reference exponent has to move (output and stored
    probabilities rescaled) in every row, for slots over batch rows and over query tiles, at block edges and remainders."""
    g = torch.Generator().manual_seed(900 + S)
    st = oracle.make_self_attention_state(g, "", C, 0, False)
    xn = torch.randn(B, S, C, generator=g).to(BF)
    pb = torch.randn(H, S, S, generator=g) + 300.0 * (torch.arange(S) // 24)[None, None, :] / max(S // 24, 1)
    pb[:, ::3] = pb[:, ::3].flip(-1)   # a third of the rows with the maximum first
    mask = (torch.rand(S, generator=g) > 0.1).float()
    r = rounded(st)
    d = C // H
    shp = (C, H, d)
    stored = (pb * 1.4426950408889634).half().float() / 1.4426950408889634   # as the kernel holds it
    ref = oracle.gated_attention(xn.float(), 1e9 * (mask[None, None, None, :] - 1), stored,
                                 r["q_projection.weight"].T.reshape(shp), r["k_projection.weight"].T.reshape(shp),
                                 r["v_projection.weight"].T.reshape(shp), r["gating_query.weight"].T.reshape(shp), None,
                                 query_b=st["q_projection.bias"].reshape(H, d))
    w = ops.PackedSelfAttention(st, "", "cuda", H)
    out = ops.attention_pair_bias_core(xn.cuda().contiguous(), w, pb.cuda().contiguous(), mask.cuda())
    ops.synchronize_and_check()
    out = out.float().cpu().reshape(B, S, H, w.Dp)[..., :d]
    assert torch.isfinite(out).all() and relf(out, ref) < 2e-2


@pytest.mark.parametrize("B,S,C,H", [(4, 65, 384, 16), (3, 33, 384, 16), (1, 129, 384, 16), (2, 1100, 384, 16), (1, 64, 768, 16),
                                     (3, 400, 768, 16)])
def test_attention_reference_exponent_moves(ops, oracle, B, S, C, H):
    """Logits of several dozen that grow along the keys: the running reference exponent has to move (output and stored
    probabilities rescaled) in every row, for slots over batch rows and over query tiles, at block edges and remainders."""
    g = torch.Generator().manual_seed(900 + S)
    st = oracle.make_self_attention_state(g, "", C, 0, False)
    xn = torch.randn(B, S, C, generator=g).to(BF)
    pb = torch.randn(H, S, S, generator=g) + 60.0 * (torch.arange(S) // 24)[None, None, :] / max(S // 24, 1)
    pb[:, ::3] = pb[:, ::3].flip(-1)   # a third of the rows with the maximum first
    mask = (torch.rand(S, generator=g) > 0.1).float()
    r = rounded(st)
    d = C // H
    shp = (C, H, d)
    ref = oracle.gated_attention(xn.float(), 1e9 * (mask[None, None, None, :] - 1), pb.half().float(),
                                 r["q_projection.weight"].T.reshape(shp), r["k_projection.weight"].T.reshape(shp),
                                 r["v_projection.weight"].T.reshape(shp), r["gating_query.weight"].T.reshape(shp), None,
                                 query_b=st["q_projection.bias"].reshape(H, d))
    w = ops.PackedSelfAttention(st, "", "cuda", H)
    out = ops.attention_pair_bias_core(xn.cuda().contiguous(), w, pb.cuda().contiguous(), mask.cuda())
    ops.synchronize_and_check()
    out = out.float().cpu().reshape(B, S, H, w.Dp)[..., :d]
    # the prepared bias is fp16 times log2(e): an absolute error of up to 0.03 in a logit near 60 * log2(e)
    assert torch.isfinite(out).all() and relf(out, ref) < 4e-2


@pytest.mark.parametrize("C,d,key", [(384, 24, 5), (384, 24, 14), (384, 24, 31), (768, 48, 62), (768, 48, 40)])
def test_attention_passes_nan_on(ops, oracle, C, d, key):
    """A key whose logits are NaN (infinite in both signs) makes every query's result NaN, whichever way its exponential is
    taken; its value row is finite."""
    g = torch.Generator().manual_seed(key)
    st = oracle.make_self_attention_state(g, "", C, 0, False)
    S, H = 70, 16
    xn = torch.randn(2, S, C, generator=g)
    xn[:, :, 0] = 0.0
    for n in ("q_projection", "k_projection", "v_projection", "gating_query"):
        st[n + ".weight"][:, 0] = 3e38 if n[0] == "k" else 0.0
    w = ops.PackedSelfAttention(st, "", "cuda", H)
    pb = torch.randn(H, S, S, generator=g).cuda()
    run = lambda: ops.attention_pair_bias_core(xn.to(BF).cuda().contiguous(), w, pb, None).float().cpu().reshape(2, S, H, w.Dp)[..., :d]
    assert torch.isfinite(run()).all()
    xn[0, key, 0] = 4.0
    out = run()
    ops.synchronize_and_check()
    assert torch.isnan(out[0]).all() and torch.isfinite(out[1]).all()


@pytest.mark.parametrize("n", [129, 137, 310])
def test_triangle_multiplication_ragged_contraction_tiles(ops, oracle, n):
    """Token counts whose last 256-wide contraction tile is mostly empty, and row counts that are no multiple of a tile."""
    g = torch.Generator().manual_seed(n)
    st = with_affine_norms(oracle.make_trimul_state(g, ""), n)
    z = torch.randn(n, n, 128, generator=g).to(BF)
    mask = (torch.rand(n, n, generator=g) > 0.2).float()
    w = ops.PackedTriMul(st, "", "cuda")
    for outgoing in (True, False):
        ref = z.float() + oracle.triangle_multiplication(rounded(st), "", z.float(), mask, outgoing)
        for _ in range(3):
            zd = z.cuda().contiguous()
            ops.triangle_multiplication_(zd, mask.cuda(), w, outgoing)
            ops.synchronize_and_check()
            check_update(z, zd, ref)


@pytest.mark.parametrize("rows", [1, 127, 129, 148 * 128, 148 * 128 + 1, 297 * 128 + 5])
def test_transition_tile_pairs(ops, oracle, rows):
    """Around the tile, the switch from one to two tiles per CTA, and an odd number of tiles."""
    g = torch.Generator().manual_seed(rows)
    st = with_affine_norms(oracle.make_transition_state(g, "", 128), rows + 1)
    x = (1.5 * torch.randn(rows, 128, generator=g) - 0.5).to(BF)
    ref = x.float() + oracle.transition(rounded(st), "", x.float())
    w = ops.PackedTransition(st, "", "cuda")
    xd = x.cuda().contiguous()
    ops.transition_(xd, w)
    ops.synchronize_and_check()
    check_update(x, xd, ref)


def test_transition_parameters_written_just_before(ops, oracle):
    """LayerNorm parameters that the kernel right before the call writes are the new ones: here the last values of a long
    projection, a kernel that lets its successor start early."""
    from distributed_xfold_b200 import _cabi
    g = torch.Generator().manual_seed(11)
    st = oracle.make_transition_state(g, "", 128)
    w = ops.PackedTransition(st, "", "cuda")
    x = torch.randn(300, 128, generator=g).to(BF)
    rows = 300_000
    src, pw = torch.randn(rows, 128, generator=g).to(BF).cuda(), (torch.randn(4, 128, generator=g) / 11).cuda()
    proj = torch.empty(4, rows, device="cuda")
    w.c.ln_gamma, w.c.ln_beta = proj[0, -128:].data_ptr(), proj[1, -128:].data_ptr()
    for _ in range(3):
        xd = x.cuda()
        proj.fill_(9.0)
        rc = _cabi.load().xfold_layernorm_fwd(_cabi.ctx(0), src.data_ptr(), 128, None, 128, rows, 128, None, None, 1e-5, 4,
                                              pw.data_ptr(), proj.data_ptr(), rows, None, None, 0, ops._stream(0))
        ops.transition_(xd, w)
        ops.synchronize_and_check()
        st["input_layer_norm.weight"], st["input_layer_norm.bias"] = proj[0, -128:].cpu(), proj[1, -128:].cpu()
        assert rc == 0 and float(proj.abs().max()) < 9.0
        r = {k: v if v.dim() == 1 else v.to(BF).float() for k, v in st.items()}
        check_update(x, xd, x.float() + oracle.transition(r, "", x.float()))


@pytest.mark.parametrize("kind", ["multiplication", "attention"])
def test_unaligned_output_weights_are_refused(ops, oracle, kind):
    """Weights that are a slice of a larger bf16 buffer, not at a multiple of 16 bytes: an error, and z as it was."""
    from distributed_xfold_b200 import _cabi
    g = torch.Generator().manual_seed(21)
    st = {k: v.to(BF).cuda() for k, v in (oracle.make_trimul_state(g, "") if kind == "multiplication" else
                                          oracle.make_grid_attention_state(g, "")).items()}
    name = "output_projection.weight"
    buf = torch.zeros(128 * 128 + 8, dtype=BF, device="cuda")
    buf[1:-7] = st[name].flatten()
    st[name] = buf[1:-7].view(128, 128)
    z = torch.randn(40, 40, 128, generator=g).to(BF).cuda()
    w = (ops.PackedTriMul if kind == "multiplication" else ops.PackedTriAttn)(st, "", "cuda")
    before = z.clone()
    with pytest.raises(_cabi.XfoldError, match="aligned"):
        (ops.triangle_multiplication_ if kind == "multiplication" else ops.triangle_attention_)(z, None, w, True)
    ops.synchronize_and_check()
    assert torch.equal(z, before)


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 148 * 128, 148 * 128 + 1])
def test_transition_one_tile_per_cta_has_the_bits_of_pairs(ops, oracle, rows):
    """Up to a tile per SM the hidden blocks take two accumulators in turn, beyond that a CTA has two tiles: the same sums in the
    same order.  The rows are the first of a call that is large enough for pairs."""
    g = torch.Generator().manual_seed(rows)
    st = oracle.make_transition_state(g, "", 128)
    w = ops.PackedTransition(st, "", "cuda")
    x = torch.randn(2 * 148 * 128 + 77, 128, generator=g).to(BF).cuda()
    want = ops.transition_(x.clone(), w)[:rows]
    got = ops.transition_(x[:rows].clone(), w)
    ops.synchronize_and_check()
    assert torch.equal(got, want)
    x = x[:min(rows, 300)].float().cpu()
    ref = x + oracle.transition(rounded(st), "", x)
    assert relf(got[:len(ref)].float().cpu(), ref) < TOL_Z
