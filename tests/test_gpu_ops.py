"""Attention / KV codec / GDN / sampling kernels vs the fp32 torch oracles."""
import math

import pytest
import torch

from ninfer_fusion_b200.ops import reference as R

pytestmark = pytest.mark.gpu

FORMATS = [("bf16", R.KV_BF16, 256), ("fp8", R.KV_FP8_ROW, 256), ("int8", R.KV_INT8_GROUP, 32),
           ("int8", R.KV_INT8_GROUP, 64), ("nvfp4", R.KV_NVFP4, 16)]


def _planes(n_pages, hkv, P, D, fmt, group):
    rb = 2 * D if fmt == R.KV_BF16 else (D // 2 if fmt == R.KV_NVFP4 else D)
    sb = {R.KV_BF16: 0, R.KV_FP8_ROW: 2, R.KV_INT8_GROUP: 2 * (D // group), R.KV_NVFP4: D // 16}[fmt]
    k = torch.zeros((n_pages, hkv, P, rb), dtype=torch.uint8, device="cuda")
    v = torch.zeros_like(k)
    ks = vs = None
    if sb:
        ks = torch.zeros((n_pages, hkv, P, sb), dtype=torch.uint8, device="cuda")
        vs = torch.zeros_like(ks)
    return k, v, ks, vs


@pytest.mark.parametrize("name,fmt,group", FORMATS)
@pytest.mark.parametrize("hq,hkv,D,P", [(6, 1, 256, 16), (24, 4, 256, 64), (16, 2, 256, 64), (8, 2, 128, 32),
                                        (3, 1, 256, 64)])
def test_prep_append_and_paged_attention(ops, name, fmt, group, hq, hkv, D, P):
    torch.manual_seed(1)
    lens = [37, 256, 1000, 300]
    B = len(lens)
    max_pages = (max(lens) + P - 1) // P
    n_pages = B * max_pages + 3
    perm = torch.randperm(n_pages)[: B * max_pages].int().view(B, max_pages).cuda()  # scattered pages
    k_codes, v_codes, k_sc, v_sc = _planes(n_pages, hkv, P, D, fmt, group)
    theta, rot = 1e7, 64
    inv_freq = R.rope_inv_freq(rot, theta).cuda()
    qw = (torch.randn(D) * 0.1).to(torch.bfloat16).cuda()
    kw = (torch.randn(D) * 0.1).to(torch.bfloat16).cuda()
    ld = (2 * hq + 2 * hkv) * D
    T = sum(lens)
    proj = torch.randn(T, ld).to(torch.bfloat16)
    # a few K outlier channels, as in the codec comparison workload
    k_off = hq * D
    for c in torch.randperm(D)[:4]:
        proj[:, k_off + c] *= 8
    proj = proj.cuda()
    tok_seq = torch.cat([torch.full((n,), b) for b, n in enumerate(lens)]).int().cuda()
    pos = torch.cat([torch.arange(n) for n in lens]).int().cuda()
    q_out = torch.empty((T, hq, D), dtype=torch.bfloat16, device="cuda")
    v_off = k_off + hkv * D + hq * D
    ops.attn_prep(proj, 0, k_off, v_off, hq, hkv, D, qw, kw, 1e-6, True, rot, inv_freq, 1.0, pos, tok_seq, pos, perm,
                  q_out, k_codes, v_codes, k_sc, v_sc, P, fmt, group, False)

    # ---- oracle for q / k / v ----
    pf = proj.float().cpu()
    qr = pf[:, : hq * D].view(T, hq, D)
    kr = pf[:, k_off:k_off + hkv * D].view(T, hkv, D)
    vr = pf[:, v_off:v_off + hkv * D].view(T, hkv, D)
    qn = R.bf16_round(R.rmsnorm(qr, qw.cpu(), 1e-6, True))
    kn = R.bf16_round(R.rmsnorm(kr, kw.cpu(), 1e-6, True))
    q_ref = R.bf16_round(R.rope_partial(qn, pos.cpu(), rot, theta))
    k_ref = R.kv_quant_dequant(R.rope_partial(kn, pos.cpu(), rot, theta), fmt, group)
    v_ref = R.kv_quant_dequant(vr, fmt, group)
    assert (q_out.float().cpu() - q_ref).abs().max().item() < 0.07

    # ---- decode-style attention: last token of each sequence + a mid-sequence query ----
    q_rows, q_seq, q_len = [], [], []
    start = 0
    for b, n in enumerate(lens):
        for p in {n - 1, n // 2}:
            q_rows.append(start + p)
            q_seq.append(b)
            q_len.append(p + 1)
        start += n
    q_rows_t = torch.tensor(q_rows).cuda()
    q = q_out[q_rows_t].contiguous()
    Tq = q.shape[0]
    gate = torch.randn(Tq, hq * D).to(torch.bfloat16).cuda()
    for split_keys, impl in ((128, 1), (512, 1), (128, 2), (512, 2)):
        if impl == 2 and D != 256:
            continue
        n_splits = (max(lens) + split_keys - 1) // split_keys
        part_o = torch.empty(Tq * hq * n_splits * D, device="cuda")
        part_ml = torch.empty(Tq * hq * n_splits * 2, device="cuda")
        out = torch.empty((Tq, hq * D), dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(q, hq, hkv, D, torch.tensor(q_seq).int().cuda(), torch.tensor(q_len).int().cuda(), perm,
                            k_codes, v_codes, k_sc, v_sc, P, fmt, group, 1 / math.sqrt(D), split_keys, n_splits,
                            part_o, part_ml, gate, out, None, None, impl, False)
        start = 0
        seq_start = [0]
        for n in lens:
            seq_start.append(seq_start[-1] + n)
        for i in range(Tq):
            b = q_seq[i]
            ks_, vs_ = k_ref[seq_start[b]:seq_start[b + 1]], v_ref[seq_start[b]:seq_start[b + 1]]
            o = R.gqa_attention(q[i:i + 1].float().cpu(), ks_, vs_, torch.tensor([q_len[i]]))
            o = R.bf16_round(o).view(-1) * torch.sigmoid(gate[i].float().cpu())
            err = (out[i].float().cpu() - o).abs().max().item()
            assert err < 0.03, f"{name} split {split_keys} impl {impl} query {i}: err {err}"


@pytest.mark.parametrize("name,fmt,group", FORMATS)
@pytest.mark.parametrize("hq,hkv", [(1, 1), (8, 1), (18, 2), (16, 1)])   # eight rows of the MMA tile, or all sixteen
@pytest.mark.parametrize("n", [1, 64, 129, 577])
def test_split_attention_group_rows(ops, name, fmt, group, hq, hkv, n):
    """The tensor-core decode kernel at the edges of its row count and of its 64-key tiles (the last key in a tile of its own,
    a second super-tile of 512 keys)."""
    torch.manual_seed(n + hq)
    D, P = 256, 16
    pages = (n + P - 1) // P
    table = torch.randperm(pages + 1)[:pages].int().view(1, pages).cuda()
    k_codes, v_codes, k_sc, v_sc = _planes(pages + 1, hkv, P, D, fmt, group)
    proj = torch.randn(n, (2 * hq + 2 * hkv) * D).to(torch.bfloat16).cuda()
    k_off, v_off = hq * D, 2 * hq * D + hkv * D
    pos, seq = torch.arange(n).int().cuda(), torch.zeros(n, dtype=torch.int32, device="cuda")
    q_all = torch.empty((n, hq, D), dtype=torch.bfloat16, device="cuda")
    ops.attn_prep(proj, 0, k_off, v_off, hq, hkv, D, None, None, 1e-6, True, 0, R.rope_inv_freq(64, 1e7).cuda(), 1.0, pos, seq,
                  pos, table, q_all, k_codes, v_codes, k_sc, v_sc, P, fmt, group, False)
    q = q_all[n - 1:].contiguous()
    out = torch.full((1, hq * D), float("nan"), dtype=torch.bfloat16, device="cuda")
    split = 640
    ops.paged_attention(q, hq, hkv, D, seq[:1], torch.tensor([n]).int().cuda(), table, k_codes, v_codes, k_sc, v_sc, P, fmt, group,
                        1 / 16, split, 1, torch.empty(hq * D, device="cuda"), torch.empty(hq * 2, device="cuda"), None, out, None,
                        None, 2, False)
    pf = proj.float().cpu()
    k_ref = R.kv_quant_dequant(pf[:, k_off:k_off + hkv * D].view(n, hkv, D), fmt, group)
    v_ref = R.kv_quant_dequant(pf[:, v_off:].view(n, hkv, D), fmt, group)
    want = R.gqa_attention(q.float().cpu(), k_ref, v_ref, torch.tensor([n]), 1 / 16).reshape(1, -1)
    # outputs are means of values: one bf16 rounding, and probabilities off by fp16 roundings of q, k, v and p and, through the
    # exponent, by the scores' own (2^-11 of the largest)
    top = float(torch.einsum("qhd,khd->hqk", q.float().cpu(), k_ref.repeat_interleave(hq // hkv, 1)).abs().max()) / 16
    tol = float(v_ref.abs().max()) * (2.0 ** -9 + 2.0 ** -10 + 2 * top * 2.0 ** -11)
    assert (out.float().cpu() - want).abs().max() <= tol


def test_paged_attention_tree_mask(ops):
    """Verify-style masks: query j sees the prefix plus the masked tree positions."""
    torch.manual_seed(3)
    hq, hkv, D, P = 6, 1, 256, 16
    L, W = 70, 5
    n_pages = 8
    table = torch.arange(n_pages).int().view(1, -1).cuda()
    k = torch.randn(L + W, hkv, D)
    v = torch.randn(L + W, hkv, D)
    k_codes, v_codes, _, _ = _planes(n_pages, hkv, P, D, R.KV_BF16, D)
    kb = k.to(torch.bfloat16).view(-1, hkv, D)
    for t in range(L + W):
        k_codes[t // P, 0, t % P] = kb[t, 0].contiguous().view(torch.uint8).cuda()
        v_codes[t // P, 0, t % P] = v.to(torch.bfloat16)[t, 0].contiguous().view(torch.uint8).cuda()
    q = torch.randn(W, hq, D).to(torch.bfloat16).cuda()
    # tree: node j sees nodes in anc[j]
    anc = [[0], [0, 1], [0, 2], [0, 1, 3], [0, 2, 4]]
    masks = torch.tensor([sum(1 << a for a in row) for row in anc], dtype=torch.long).cuda()
    base = torch.full((W,), L, dtype=torch.int32).cuda()
    out = torch.empty((W, hq * D), dtype=torch.bfloat16, device="cuda")
    part_o = torch.empty(W * hq * D, device="cuda")
    part_ml = torch.empty(W * hq * 2, device="cuda")
    vis = torch.zeros(W, L + W, dtype=torch.bool)
    vis[:, :L] = True
    for j, row in enumerate(anc):
        for a in row:
            vis[j, L + a] = True
    ref = R.gqa_attention(q.float().cpu(), R.bf16_round(k), R.bf16_round(v), None, 1 / 16, vis).reshape(W, -1)
    for impl in (1, 2):
        out.zero_()
        ops.paged_attention(q, hq, hkv, D, torch.zeros(W).int().cuda(), torch.full((W,), L + W).int().cuda(), table,
                            k_codes, v_codes, None, None, P, R.KV_BF16, D, 1 / 16, 128, 1, part_o, part_ml, None, out,
                            masks, base, impl, False)
        assert (out.float().cpu() - ref).abs().max().item() < 0.02, f"impl {impl}"
    vis = torch.zeros(W, L + W, dtype=torch.bool)
    vis[:, :L] = True
    for j, row in enumerate(anc):
        for a in row:
            vis[j, L + a] = True
    ref = R.gqa_attention(q.float().cpu(), R.bf16_round(k), R.bf16_round(v), None, 1 / 16, vis).reshape(W, -1)
    assert (out.float().cpu() - ref).abs().max().item() < 0.02


@pytest.mark.parametrize("heads", [(2, 6), (4, 16), (8, 32), (16, 48)])  # row-split over 8 / 4 / 2 / 1 CTAs per head
@pytest.mark.parametrize("lens", [[1, 1, 1], [5, 1, 17], [64, 3], [300, 40]])
def test_conv_and_gdn_recurrent(ops, lens, heads):
    torch.manual_seed(2)
    (hk, hv), d = heads, 128
    qk, vd = hk * d, hv * d
    C = 2 * qk + vd
    ld = C + vd + 2 * hv
    T, B = sum(lens), len(lens)
    proj = (torch.randn(T, ld) * 0.7).to(torch.bfloat16)
    conv_w = (torch.randn(C, 4) * 0.3).to(torch.bfloat16)
    A_log = torch.rand(hv) * 2 - 1
    dt_bias = torch.rand(hv) * 2 - 1.5
    nw = (1 + 0.1 * torch.randn(d)).to(torch.bfloat16)
    slots = [3, 0, 2][:B]
    n_slots = 4
    conv_state = (torch.randn(n_slots, 3, C) * 0.5).to(torch.bfloat16)
    ssm = torch.randn(n_slots, hv, d, d) * 0.1
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    tok_seq = torch.cat([torch.full((n,), b) for b, n in enumerate(lens)]).int()

    conv_state_g, ssm_g = conv_state.clone().cuda(), ssm.clone().cuda()
    conv_out = torch.empty((T, C), dtype=torch.bfloat16, device="cuda")
    ops.causal_conv1d_silu(proj.cuda(), 0, C, conv_w.cuda(), cu.cuda(), tok_seq.cuda(), torch.tensor(slots).int().cuda(),
                           conv_state_g, conv_out, True, all(n == 1 for n in lens), False)
    out = torch.empty((T, vd), dtype=torch.bfloat16, device="cuda")
    ops.gdn_recurrent(conv_out, 0, qk, 2 * qk, proj.cuda(), C, C + vd, C + vd + hv, hk, hv, A_log.cuda(),
                      dt_bias.cuda(), nw.cuda(), 1e-6, cu.cuda(), torch.tensor(slots).int().cuda(), ssm_g, True, out,
                      False)
    # verify pass must leave the state untouched
    ssm_v = ssm.clone().cuda()
    out_v = torch.empty_like(out)
    ops.gdn_recurrent(conv_out, 0, qk, 2 * qk, proj.cuda(), C, C + vd, C + vd + hv, hk, hv, A_log.cuda(),
                      dt_bias.cuda(), nw.cuda(), 1e-6, cu.cuda(), torch.tensor(slots).int().cuda(), ssm_v, False,
                      out_v, False)
    assert torch.equal(ssm_v.cpu(), ssm) and torch.equal(out_v, out)
    if all(n == 1 for n in lens):
        # decode: the same step with the convolution inside the recurrent kernel gives the same bits and the same
        # history as the two launches above
        conv_f, ssm_f = conv_state.clone().cuda(), ssm.clone().cuda()
        out_f = torch.full_like(out, float("nan"))
        ops.gdn_recurrent(proj.cuda(), 0, qk, 2 * qk, proj.cuda(), C, C + vd, C + vd + hv, hk, hv, A_log.cuda(),
                          dt_bias.cuda(), nw.cuda(), 1e-6, cu.cuda(), torch.tensor(slots).int().cuda(), ssm_f, True, out_f,
                          False, None, None, None, conv_w.cuda(), conv_f)
        assert torch.equal(out_f, out) and torch.equal(ssm_f, ssm_g) and torch.equal(conv_f, conv_state_g)

    for b, n in enumerate(lens):
        s, e = int(cu[b]), int(cu[b + 1])
        pj = proj[s:e].float()
        cref, new_conv = R.causal_conv1d_silu(pj[:, :C], conv_w, conv_state[slots[b]])
        cref = R.bf16_round(cref)
        assert (conv_out[s:e].float().cpu() - cref).abs().max().item() < 0.02
        assert torch.equal(conv_state_g[slots[b]].cpu(), new_conv.to(torch.bfloat16))
        q = cref[:, :qk].view(n, hk, d)
        k = cref[:, qk:2 * qk].view(n, hk, d)
        v = cref[:, 2 * qk:].view(n, hv, d)
        z = pj[:, C:C + vd].view(n, hv, d)
        g, beta = R.gdn_gating(pj[:, C + vd:C + vd + hv], pj[:, C + vd + hv:], A_log, dt_bias)
        o, new_s = R.gdn_recurrent(q, k, v, g, beta, ssm[slots[b]])
        y = R.gated_rmsnorm(R.bf16_round(o), z, nw).view(n, vd)
        err = (out[s:e].float().cpu() - y).abs().max().item()
        assert err < 0.05 * max(1.0, y.abs().max().item()), f"seq {b} err {err}"
        assert (ssm_g[slots[b]].cpu() - new_s).abs().max().item() < 2e-3 * max(1.0, new_s.abs().max().item())
    untouched = [s for s in range(n_slots) if s not in slots]
    for s in untouched:
        assert torch.equal(ssm_g[s].cpu(), ssm[s])


@pytest.mark.parametrize("lens", [[64], [16, 16, 32], [1, 3, 60, 200], [79], [130, 2, 1, 1]])
def test_conv_runs_match_single_tokens(ops, lens):
    """The kernel for runs of tokens (two channels an instruction, quotient by residual) against the per-token one, which takes
    steps of fewer than 64 tokens and divides: the same bits, infinities, NaN, large and tiny values among them."""
    torch.manual_seed(6)
    T, B, C = sum(lens), len(lens), 1032
    x = torch.randn(T, C + 8).bfloat16()
    for k, v in enumerate((float("inf"), float("-inf"), float("nan"), 3e38, -3e38, -1000.0, 1000.0, -87.5, -89.0, 1e-38, -1e-38, -0.0)):
        x[(7 * k + 3) % T, k::101] = v
    x = x.cuda()
    w = (torch.randn(C, 4) * 0.5).bfloat16().cuda()
    hist = torch.randn(B, 3, C).bfloat16().cuda()
    slot = torch.randperm(B).int().cuda()
    tok = torch.cat([torch.full((n,), b) for b, n in enumerate(lens)]).int().cuda()
    cu = torch.tensor([0] + lens).cumsum(0).int().cuda()
    want_hist, got_hist = hist.clone(), hist.clone()
    got = torch.full((T, C), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.causal_conv1d_silu(x, 0, C, w, cu, tok, slot, got_hist, got, True, False, True)
    want = torch.empty_like(got)
    for b, n in enumerate(lens):
        for o in range(0, n, 48):
            m, s = min(48, n - o), int(cu[b]) + o
            out = torch.empty((m, C), dtype=torch.bfloat16, device="cuda")
            ops.causal_conv1d_silu(x[s:s + m], 0, C, w, torch.tensor([0, m]).int().cuda(), torch.zeros(m).int().cuda(), slot[b:b + 1],
                                   want_hist, out, True, False, False)
            want[s:s + m] = out
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(5.0), want.nan_to_num(5.0))
    assert torch.equal(got_hist.view(torch.int16), want_hist.view(torch.int16))


@pytest.mark.parametrize("heads", [(16, 48), (16, 32)])
@pytest.mark.parametrize("pdl", [False, True])
@pytest.mark.parametrize("ragged", [False, True])
def test_gdn_step_of_many_states(ops, heads, pdl, ragged):
    """Enough states for the streaming kernel, the last round of a part of the CTAs; `commit` of ones takes the general kernel.
    Ragged: as many tokens as sequences, but sequences of none and of several."""
    torch.manual_seed(3)
    (hk, hv), d = heads, 128
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B = -(-13 * sms // (2 * hv)) + 1
    qk, vd = hk * d, hv * d
    C = 2 * qk + vd
    ld = C + vd + 2 * hv
    conv = torch.randn(B, C, device="cuda").to(torch.bfloat16)
    proj = torch.randn(B, ld, device="cuda").to(torch.bfloat16)
    A_log, dt_bias = torch.rand(hv, device="cuda") * 2 - 1, torch.rand(hv, device="cuda") * 2 - 1.5
    nw = (1 + 0.1 * torch.randn(d, device="cuda")).to(torch.bfloat16)
    lens = [1] * B
    if ragged:
        lens[0], lens[1], lens[5], lens[6], lens[7], lens[B - 1] = 0, 2, 0, 3, 0, 1
        assert sum(lens) == B
    cu = torch.tensor([0] + lens, device="cuda").cumsum(0).int()
    slot = torch.randperm(B + 1, device="cuda")[:B].int()
    states = torch.randn(B + 1, hv, d, d, device="cuda") * 0.2
    got = []
    for commit in (torch.ones(B, dtype=torch.uint8, device="cuda"), None):
        s, out = states.clone(), torch.full((B, vd), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.gdn_recurrent(conv, 0, qk, 2 * qk, proj, C, C + vd, C + vd + hv, hk, hv, A_log, dt_bias, nw, 1e-6, cu, slot, s, True, out,
                          pdl, None, commit)
        got.append((s, out))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert not got[1][1].isnan().any() and not torch.equal(got[1][0], states)


@pytest.mark.parametrize("heads", [(16, 48), (16, 32)])
def test_gdn_step_of_many_states_quantises_its_rows(ops, status, heads):
    """The streaming step's rows as the next product's nvfp4 operand: codes and scales of the general kernel (`commit` of ones), and
    those of the quantiser over the step's output."""
    torch.manual_seed(4)
    (hk, hv), d = heads, 128
    B = -(-13 * torch.cuda.get_device_properties(0).multi_processor_count // (2 * hv)) + 1
    qk, vd = hk * d, hv * d
    C = 2 * qk + vd
    conv = torch.randn(B, C, device="cuda").to(torch.bfloat16)
    proj = torch.randn(B, C + vd + 2 * hv, device="cuda").to(torch.bfloat16)
    A_log, dt_bias = torch.rand(hv, device="cuda") * 2 - 1, torch.rand(hv, device="cuda") * 2 - 1.5
    nw = (1 + 0.1 * torch.randn(d, device="cuda")).to(torch.bfloat16)
    cu, slot = torch.arange(B + 1, device="cuda").int(), torch.randperm(B, device="cuda").int()
    states = torch.randn(B, hv, d, d, device="cuda") * 0.2
    size = int(ops.nvfp4_act_scale_bytes(B, vd))
    got = []
    for commit in (torch.ones(B, dtype=torch.uint8, device="cuda"), None):
        out = torch.full((B, vd), float("nan"), dtype=torch.bfloat16, device="cuda")
        codes, plane = torch.full((B, vd // 2), 255, dtype=torch.uint8, device="cuda"), torch.zeros(size, dtype=torch.uint8, device="cuda")
        ops.gdn_recurrent(conv, 0, qk, 2 * qk, proj, C, C + vd, C + vd + hv, hk, hv, A_log, dt_bias, nw, 1e-6, cu, slot, states.clone(),
                          True, out, True, None, commit, None, None, None, codes, plane, status.tensor)
        got.append((out, codes, plane))
    codes, plane = torch.empty_like(got[0][1]), torch.zeros_like(got[0][2])
    ops.quant_act_nvfp4(got[0][0], codes, plane)
    for a, b in zip(*got):
        assert torch.equal(a, b)
    assert torch.equal(got[1][1], codes) and torch.equal(got[1][2], plane)
    status.check("streaming step")


@pytest.mark.parametrize("T", [9, 200])
def test_embed_rmsnorm(ops, T):
    torch.manual_seed(0)
    V, N = 1000, 5120
    table = torch.randn(V, N).to(torch.bfloat16).cuda()
    ids = torch.randint(0, V, (T,)).int().cuda()
    x = torch.empty((T, N), dtype=torch.bfloat16, device="cuda")
    ops.embed_gather(ids, table, x, False)
    assert torch.equal(x, table[ids.long()])
    w = (torch.randn(N) * 0.1).to(torch.bfloat16).cuda()
    delta = torch.randn(T, N).to(torch.bfloat16).cuda()
    r_out = torch.empty_like(x)
    normed = torch.empty_like(x)
    ops.add_rmsnorm(None, 0, delta, x, r_out, w, normed, T, N, 1e-6, True, False)
    xr = (x.float() + delta.float()).to(torch.bfloat16)
    assert torch.equal(r_out, xr)
    ref = R.rmsnorm(xr.float().cpu(), w.cpu(), 1e-6, True)
    assert (normed.float().cpu() - ref).abs().max().item() < 0.05


def test_argmax_and_sampling(ops):
    torch.manual_seed(0)
    T, V = 5, 248320
    logits = torch.randn(T, V).to(torch.bfloat16).cuda()
    logits[1, 77] = 50.0
    logits[1, 99999] = 50.0  # tie -> lowest id
    out = torch.empty(T, dtype=torch.int32, device="cuda")
    ops.argmax_rows(logits, out, False)
    assert torch.equal(out.cpu(), R.argmax_lowest(logits.cpu()))
    assert int(out[1]) == 77
    # greedy through the sampler (temperature 0) must agree with arg-max
    temp = torch.zeros(T, device="cuda")
    out2 = torch.empty_like(out)
    ops.sample_rows(logits, temp, None, None, None, None, None, None, None, None, 0, out2, None)
    assert torch.equal(out, out2)
    # stochastic: draws stay inside the top-k set, are reproducible per (seed, position), vary with position
    temp = torch.ones(T, device="cuda")
    top_k = torch.full((T,), 5, dtype=torch.int32, device="cuda")
    seeds = torch.arange(T, dtype=torch.int64, device="cuda") + 11
    posn = torch.arange(T, dtype=torch.int32, device="cuda")
    a = torch.empty_like(out)
    b = torch.empty_like(out)
    ops.sample_rows(logits, temp, top_k, None, None, None, None, None, seeds, posn, 0, a, None)
    ops.sample_rows(logits, temp, top_k, None, None, None, None, None, seeds, posn, 0, b, None)
    assert torch.equal(a, b)
    top5 = logits.float().topk(5, dim=-1).indices
    for t in range(T):
        assert int(a[t]) in top5[t].tolist()
    # top_p tiny -> always the arg-max
    top_p = torch.full((T,), 1e-4, device="cuda")
    ops.sample_rows(logits, temp, top_k, top_p, None, None, None, None, seeds, posn, 0, b, None)
    assert torch.equal(b, out)
    # distribution check on a 3-way row
    row = torch.full((1, 64), -30.0)
    row[0, 3], row[0, 10], row[0, 20] = 2.0, 1.0, 0.0
    row = row.to(torch.bfloat16).cuda().repeat(4096, 1)
    seeds = torch.arange(4096, dtype=torch.int64, device="cuda")
    draws = torch.empty(4096, dtype=torch.int32, device="cuda")
    ops.sample_rows(row, torch.ones(4096, device="cuda"), None, None, None, None, None, None, seeds, None, 0, draws, None)
    p = torch.softmax(torch.tensor([2.0, 1.0, 0.0]), 0)
    freq = torch.tensor([(draws == i).float().mean().item() for i in (3, 10, 20)])
    assert (freq - p).abs().max().item() < 0.03


def test_speculative_accept(ops):
    target = torch.tensor([[5, 6, 7, 8], [5, 6, 7, 8], [1, 2, 3, 4]], dtype=torch.int32)
    draft = torch.tensor([[5, 6, 7], [5, 9, 7], [0, 2, 3]], dtype=torch.int32)
    n_ref, out_ref = R.accept_greedy_chain(target, draft)
    n = torch.empty(3, dtype=torch.int32, device="cuda")
    out = torch.empty((3, 4), dtype=torch.int32, device="cuda")
    ops.accept_greedy_chain(target.cuda(), draft.cuda(), n, out)
    assert torch.equal(n.cpu(), n_ref) and torch.equal(out.cpu(), out_ref)
    # tree: 0 -> {1, 2}; 1 -> {3}; 2 -> {4}; 3 -> {5}
    parent = torch.tensor([[-1, 0, 0, 1, 2, 3]], dtype=torch.int32)
    tok = torch.tensor([[0, 11, 12, 13, 14, 15]], dtype=torch.int32)
    tgt = torch.tensor([[12, 13, 14, 15, 99, 98]], dtype=torch.int32)  # accepts 2 then 4
    nr, tr, nodes_r = R.accept_greedy_tree(tgt, tok, parent, 4)
    n1 = torch.empty(1, dtype=torch.int32, device="cuda")
    t1 = torch.empty((1, 5), dtype=torch.int32, device="cuda")
    nd = torch.empty((1, 5), dtype=torch.int32, device="cuda")
    ops.accept_greedy_tree(tgt.cuda(), tok.cuda(), parent.cuda(), 4, n1, t1, nd)
    assert torch.equal(n1.cpu(), nr) and torch.equal(t1.cpu(), tr) and torch.equal(nd.cpu(), nodes_r)
    assert int(nr[0]) == 2 and tr[0, :3].tolist() == [12, 14, 99]


@pytest.mark.parametrize("name,fmt,group", FORMATS)
@pytest.mark.parametrize("hq,hkv", [(6, 1), (24, 4), (16, 2), (3, 1)])
def test_prefill_attention(ops, name, fmt, group, hq, hkv):
    """Causal block attention over a ragged chunk (one sequence continues mid-way) vs the fp32 oracle."""
    torch.manual_seed(4)
    D, P = 256, 16
    lens = [150, 37]
    chunk_from = [60, 0]            # tokens [60, 150) of sequence 0 and all of sequence 1 are the "chunk"
    B = len(lens)
    max_pages = (max(lens) + P - 1) // P
    n_pages = B * max_pages + 2
    table = torch.randperm(n_pages)[: B * max_pages].int().view(B, max_pages).cuda()
    k_codes, v_codes, k_sc, v_sc = _planes(n_pages, hkv, P, D, fmt, group)
    inv_freq = R.rope_inv_freq(64, 1e7).cuda()
    ld = (2 * hq + 2 * hkv) * D
    T = sum(lens)
    proj = torch.randn(T, ld).to(torch.bfloat16).cuda()
    tok_seq = torch.cat([torch.full((n,), b) for b, n in enumerate(lens)]).int().cuda()
    pos = torch.cat([torch.arange(n) for n in lens]).int().cuda()
    q_all = torch.empty((T, hq, D), dtype=torch.bfloat16, device="cuda")
    k_off, v_off = hq * D, hq * D + hkv * D + hq * D
    ops.attn_prep(proj, 0, k_off, v_off, hq, hkv, D, None, None, 1e-6, True, 0, inv_freq, 1.0, pos, tok_seq, pos, table,
                  q_all, k_codes, v_codes, k_sc, v_sc, P, fmt, group, False)
    # the chunk's tokens
    rows, starts = [], [0, lens[0]]
    for b in range(B):
        rows += list(range(starts[b] + chunk_from[b], starts[b] + lens[b]))
    rows_t = torch.tensor(rows).cuda()
    q = q_all[rows_t].contiguous()
    q_seq = tok_seq[rows_t].contiguous()
    kv_len = (pos[rows_t] + 1).contiguous()
    gate = torch.randn(len(rows), hq * D).to(torch.bfloat16).cuda()
    qt = int(ops.prefill_attn_block_tokens(hq, hkv))
    blk_s, blk_c, t = [], [], 0
    for b in range(B):
        n = lens[b] - chunk_from[b]
        for o in range(0, n, qt):
            blk_s.append(t + o)
            blk_c.append(min(qt, n - o))
        t += n
    out = torch.full((len(rows), hq * D), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.paged_attention_prefill(q, hq, hkv, D, q_seq, kv_len, torch.tensor(blk_s).int().cuda(),
                                torch.tensor(blk_c).int().cuda(), table, k_codes, v_codes, k_sc, v_sc, P, fmt, group,
                                1 / 16, gate, out, False)
    pf = proj.float().cpu()
    k_ref = R.kv_quant_dequant(pf[:, k_off:k_off + hkv * D].view(T, hkv, D), fmt, group)
    v_ref = R.kv_quant_dequant(pf[:, v_off:v_off + hkv * D].view(T, hkv, D), fmt, group)
    worst = 0.0
    for i, r in enumerate(rows):
        b = int(tok_seq[r])
        ks_, vs_ = k_ref[starts[b]:starts[b] + lens[b]], v_ref[starts[b]:starts[b] + lens[b]]
        o = R.gqa_attention(q[i:i + 1].float().cpu(), ks_, vs_, torch.tensor([int(kv_len[i])]), 1 / 16)
        o = R.bf16_round(o).reshape(-1) * torch.sigmoid(gate[i].float().cpu())
        worst = max(worst, (out[i].float().cpu() - o).abs().max().item())
    assert worst < 0.03, f"{name}: err {worst}"


@pytest.mark.parametrize("name,fmt,group", FORMATS)
@pytest.mark.parametrize("hq,hkv,n,T", [(2, 2, 1, 1), (24, 4, 63, 63), (24, 4, 64, 3), (24, 4, 65, 65), (128, 1, 129, 3),
                                        (16, 2, 191, 40), (6, 1, 200, 200), (24, 4, 1100, 30)])
def test_prefill_attention_tile_edges(ops, status, name, fmt, group, hq, hkv, n, T):
    """The last T of n positions at the edges of the 64-key tiles, groups from one head to all 128 rows: keys that grow along
    the sequence (a row's frame moves in most tiles), values so large that fp8 rows have scales above 1024, a gate whose rows
    start at any even element."""
    torch.manual_seed(n)
    D, P = 256, 16
    pages = (n + P - 1) // P
    table = torch.randperm(pages + 1)[:pages].int().view(1, pages).cuda()
    k_codes, v_codes, k_sc, v_sc = _planes(pages + 1, hkv, P, D, fmt, group)
    big = 2e5 if name == "fp8" else 1.0
    proj = torch.randn(n, (2 * hq + 2 * hkv) * D)
    k_off, v_off = hq * D, 2 * hq * D + hkv * D
    proj[:, k_off:k_off + hkv * D] *= (0.2 + 2.0 * torch.arange(n) / n)[:, None]
    proj[:, v_off:] *= big
    proj = proj.to(torch.bfloat16).cuda()
    pos, seq = torch.arange(n).int().cuda(), torch.zeros(n, dtype=torch.int32, device="cuda")
    q_all = torch.empty((n, hq, D), dtype=torch.bfloat16, device="cuda")
    ops.attn_prep(proj, 0, k_off, v_off, hq, hkv, D, None, None, 1e-6, True, 0, R.rope_inv_freq(64, 1e7).cuda(), 1.0, pos, seq,
                  pos, table, q_all, k_codes, v_codes, k_sc, v_sc, P, fmt, group, False)
    q = q_all[n - T:].contiguous()
    gate = torch.randn(T, hq * D + 6).to(torch.bfloat16).cuda()[:, 2:2 + hq * D]
    qt = int(ops.prefill_attn_block_tokens(hq, hkv))
    starts = list(range(0, T, qt))
    out = torch.full((T, hq * D), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.paged_attention_prefill(q, hq, hkv, D, seq[n - T:].contiguous(), (pos[n - T:] + 1).contiguous(), torch.tensor(starts).int().cuda(),
                                torch.tensor([min(qt, T - o) for o in starts]).int().cuda(), table, k_codes, v_codes, k_sc, v_sc, P,
                                fmt, group, 1 / 16, gate, out, False, 0, None, status.tensor)
    pf = proj.float().cpu()
    k_ref = R.kv_quant_dequant(pf[:, k_off:k_off + hkv * D].view(n, hkv, D), fmt, group)
    v_ref = R.kv_quant_dequant(pf[:, v_off:].view(n, hkv, D), fmt, group)
    o = R.gqa_attention(q.float().cpu(), k_ref, v_ref, torch.arange(n - T, n) + 1, 1 / 16)
    want = o.reshape(T, -1) * torch.sigmoid(gate.float().cpu())
    # outputs are means of values: bf16 roundings before and after the gate, and probabilities off by fp16 roundings of
    # q, k, v and p and, through the exponent, by the scores' own (2^-11 of the largest)
    top = float(torch.einsum("qhd,khd->hqk", q.float().cpu(), k_ref.repeat_interleave(hq // hkv, 1)).abs().max()) / 16
    tol = float(v_ref.abs().max()) * (2.0 ** -8 + 2.0 ** -10 + 2 * top * 2.0 ** -11)
    assert (out.float().cpu() - want).abs().max() <= tol
    status.check("prefill attention")


@pytest.mark.parametrize("hq,hkv", [(1, 1), (6, 2), (24, 4), (8, 1)])
@pytest.mark.parametrize("P,window,tree", [(64, 0, False), (7, 0, True), (48, 100, False), (160, 300, False)])
def test_nvfp4_decode_attention_of_aligned_scales(ops, hq, hkv, P, window, tree):
    """Row scales at a 16-byte boundary are read sixteen at once, by a kernel whose products and sums are those of the general
    one, which takes scales at any address (and splits of fewer than four tiles): the same bits, for any page size, released pages,
    windows, tree masks and lengths at the edges of tiles and splits."""
    torch.manual_seed(P)
    D, lens, split, ns = 256, [1, 63, 64, 65, 257, 700, 256, 511], 256, 3
    B, pages = len(lens), (max(lens) + P - 1) // P
    table = torch.randperm(B * pages + 1)[: B * pages].int().view(B, pages).cuda()
    k, v, ks, vs = _planes(B * pages + 1, hkv, P, D, R.KV_NVFP4, 16)
    for codes, scales in ((k, ks), (v, vs)):
        codes.copy_(torch.randint(0, 256, codes.shape, dtype=torch.uint8))
        scales.copy_(torch.randint(0, 0x7f, scales.shape, dtype=torch.uint8))
    if window:
        for b, n in enumerate(lens):
            table[b, : max(0, n - window) // P] = -1
    elsewhere = torch.empty(ks.numel() + 16, dtype=torch.uint8, device="cuda")[8:8 + ks.numel()].view(ks.shape)
    elsewhere.copy_(ks)
    q = torch.randn(B, hq, D).to(torch.bfloat16).cuda()
    kv_len, seq = torch.tensor(lens).int().cuda(), torch.arange(B).int().cuda()
    seq[2] = -1
    mask = torch.randint(0, 2 ** 62, (B,)).cuda() if tree else None
    base = (kv_len - 60).clamp(min=0).int() if tree else None
    got = []
    for scales in (ks, elsewhere):
        po, pm = torch.zeros(B * hq * ns * D, device="cuda"), torch.zeros(B * hq * ns * 2, device="cuda")
        out = torch.full((B, hq * D), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(q, hq, hkv, D, seq, kv_len, table, k, v, scales, vs, P, R.KV_NVFP4, 16, 1 / 16, split, ns, po, pm, None,
                            out, mask, base, 2, False, window)
        got.append((po, pm, out))
    for a, b in zip(*got):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    assert got[0][1].isfinite().any() and not got[0][2].isnan().any()


@pytest.mark.parametrize("name,fmt,group", FORMATS)
def test_prefill_attention_does_not_depend_on_pages(ops, status, name, fmt, group):
    """The same rows in pages of a tile, of sizes that neither divide a tile nor are divided by one, and with the pages behind a
    window released: the same bits, with the window and without."""
    torch.manual_seed(9)
    D, hq, hkv, n, T = 256, 6, 2, 333, 70
    ld, k_off, v_off = (2 * hq + 2 * hkv) * D, hq * D, 2 * hq * D + hkv * D
    proj = torch.randn(n, ld).to(torch.bfloat16).cuda()
    pos, seq = torch.arange(n).int().cuda(), torch.zeros(n, dtype=torch.int32, device="cuda")
    qt = int(ops.prefill_attn_block_tokens(hq, hkv))
    starts = list(range(0, T, qt))
    counts = torch.tensor([min(qt, T - o) for o in starts]).int().cuda()
    outs = {}
    for P in (64, 7, 48, 160):
        pages = (n + P - 1) // P
        table = torch.randperm(pages + 1)[:pages].int().view(1, pages).cuda()
        planes = _planes(pages + 1, hkv, P, D, fmt, group)
        q = torch.empty((n, hq, D), dtype=torch.bfloat16, device="cuda")
        ops.attn_prep(proj, 0, k_off, v_off, hq, hkv, D, None, None, 1e-6, True, 0, R.rope_inv_freq(64, 1e7).cuda(), 1.0, pos,
                      seq, pos, table, q, *planes, P, fmt, group, False)
        for window, released in ((0, 0), (100, 0), (100, (n - T + 1 - 100) // P)):
            used = table.clone()
            used[:, :released] = -1
            out = torch.full((T, hq * D), float("nan"), dtype=torch.bfloat16, device="cuda")
            ops.paged_attention_prefill(q[n - T:].contiguous(), hq, hkv, D, seq[:T], (pos[n - T:] + 1).contiguous(),
                                        torch.tensor(starts).int().cuda(), counts, used, *planes, P, fmt, group, 1 / 16, None, out,
                                        False, window, None, status.tensor)
            assert torch.equal(out, outs.setdefault(window, out)), (P, window, released)
    assert not outs[0].isnan().any() and not torch.equal(outs[0], outs[100])
    status.check("prefill attention")


@pytest.mark.parametrize("name,fmt,group", FORMATS)
def test_prefill_attention_halves_of_a_row(ops, status, name, fmt, group):
    """The two warps of a row store probabilities over each other's scores.  Scores that grow from tile to tile in one part of the
    rows and not in the other, on all SMs at once: every run gives the same bits, and those of the queries by themselves."""
    torch.manual_seed(11)
    D, hq, hkv, n, T, P = 256, 8, 2, 1100, 600, 64
    ld, k_off, v_off = (2 * hq + 2 * hkv) * D, hq * D, 2 * hq * D + hkv * D
    proj = torch.randn(n, ld)
    proj[:, k_off:k_off + hkv * D] *= torch.linspace(0.2, 3.0, n)[:, None]
    proj[::3, :hq * D] *= -1
    proj = proj.to(torch.bfloat16).cuda()
    pos, seq = torch.arange(n).int().cuda(), torch.zeros(n, dtype=torch.int32, device="cuda")
    pages = (n + P - 1) // P
    table = torch.randperm(pages)[:pages].int().view(1, pages).cuda()
    planes = _planes(pages, hkv, P, D, fmt, group)
    q = torch.empty((n, hq, D), dtype=torch.bfloat16, device="cuda")
    ops.attn_prep(proj, 0, k_off, v_off, hq, hkv, D, None, None, 1e-6, True, 0, R.rope_inv_freq(64, 1e7).cuda(), 1.0, pos, seq, pos,
                  table, q, *planes, P, fmt, group, False)
    qt = int(ops.prefill_attn_block_tokens(hq, hkv))

    def run(first, count):
        starts = list(range(0, count, qt))
        out = torch.full((count, hq * D), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.paged_attention_prefill(q[first:first + count].contiguous(), hq, hkv, D, seq[:count], (pos[first:first + count] + 1).contiguous(),
                                    torch.tensor(starts).int().cuda(), torch.tensor([min(qt, count - o) for o in starts]).int().cuda(),
                                    table, *planes, P, fmt, group, 1 / 16, None, out, False, 0, None, status.tensor)
        return out
    first = run(n - T, T)
    assert not first.isnan().any()
    for _ in range(6):
        assert torch.equal(run(n - T, T), first)
    for at in (n - T, n - T + 333, n - 2):
        assert torch.equal(run(at, 2), first[at - n + T:at - n + T + 2])
    status.check("prefill attention")


def test_prefill_attention_largest_key_weighs_one(ops, status):
    """The 64 keys of the first tile score 0, one key of the second 2.03125 (in powers of two): that key's probability against
    the row's largest score is one, exactly, so outputs are its value times an fp32 factor.  Against the first tile's frame it
    would be 2^2.03125, which fp16 holds 4e-4 too small: every fourth output would round the other way."""
    H, D, P, n = 8, 256, 64, 128
    table = torch.arange(2).int().view(1, 2).cuda()
    k, v, _, _ = _planes(2, H, P, D, R.KV_BF16, 256)
    k.view(torch.bfloat16)[1, :, 0, 0] = 2.03125
    val = torch.randn(H, D, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16)
    v.view(torch.bfloat16)[1, :, 0] = val.cuda()
    q = torch.zeros((1, H, D), dtype=torch.bfloat16, device="cuda")
    q[:, :, 0] = 1.0
    out = torch.empty((1, H * D), dtype=torch.bfloat16, device="cuda")
    one = torch.ones(1, dtype=torch.int32, device="cuda")
    ops.paged_attention_prefill(q, H, H, D, 0 * one, n * one, 0 * one, one, table, k, v, None, None, P, R.KV_BF16, 256,
                                1 / 1.4426950408889634, None, out, False, 0, None, status.tensor)
    want = (val.double() / (1 + 127 * 2.0 ** -2.03125)).to(torch.bfloat16).view(1, -1)
    # a handful of fp32 roundings (1e-6 of a value) moves an output across a bf16 tie in one of some 4000 cases
    assert (out.cpu() != want).sum() <= 4
    status.check("largest key")


def test_stochastic_draft_verification_preserves_the_target_distribution(ops):
    """Deterministic drafts verified by speculative sampling: accept w.p. p(draft), else draw from p without the
    draft.  Over many seeds the emitted token must follow p itself and the acceptance rate must be p(draft)."""
    torch.manual_seed(0)
    V, n = 64, 6000
    base = torch.randn(V) * 1.5
    logits = base.to(torch.bfloat16)[None].repeat(n, 1).contiguous().cuda()
    k = 8
    vals, idx = torch.sort(logits[0].float().cpu(), descending=True, stable=True)
    p = torch.softmax(vals[:k], 0)                    # temperature 1, top-k 8, no top-p
    draft_tok = int(idx[2])                           # third most likely token, p ~ p[2]
    temp = torch.ones(n, device="cuda")
    topk = torch.full((n,), k, dtype=torch.int32, device="cuda")
    seeds = torch.arange(n, dtype=torch.int64, device="cuda")
    pos = torch.full((n,), 17, dtype=torch.int32, device="cuda")
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    acc = torch.empty(n, dtype=torch.int32, device="cuda")
    drafts = torch.full((n,), draft_tok, dtype=torch.int32, device="cuda")
    ops.sample_rows(logits, temp, topk, None, None, None, None, None, seeds, pos, 0, out, None, drafts, acc)
    rate = acc.float().mean().item()
    assert abs(rate - p[2].item()) < 0.02
    assert bool((out[acc.bool()] == draft_tok).all()) and bool((out[~acc.bool()] != draft_tok).all())
    emp = torch.bincount(out.cpu().long(), minlength=V).float() / n
    want = torch.zeros(V)
    want[idx[:k]] = p
    assert (emp - want).abs().max().item() < 0.025
    # a draft outside the candidate set is always rejected; a greedy row accepts only the arg-max
    drafts.fill_(int(idx[-1]))
    ops.sample_rows(logits, temp, topk, None, None, None, None, None, seeds, pos, 0, out, None, drafts, acc)
    assert acc.sum().item() == 0
    temp.zero_()
    drafts.fill_(int(idx[0]))
    ops.sample_rows(logits, temp, topk, None, None, None, None, None, seeds, pos, 0, out, None, drafts, acc)
    assert acc.sum().item() == n and bool((out == int(idx[0])).all())
    # chain acceptance on top: rows of one sequence are columns of the verify window
    B, K = 4, 3
    lg = logits[: B * (K + 1)]
    temp = torch.ones(B * (K + 1), device="cuda")
    d = torch.full((B, K + 1), -1, dtype=torch.int32, device="cuda")
    d[:, :K] = draft_tok
    tok = torch.empty(B * (K + 1), dtype=torch.int32, device="cuda")
    ok = torch.empty(B * (K + 1), dtype=torch.int32, device="cuda")
    ops.sample_rows(lg, temp, topk[: B * (K + 1)], None, None, None, None, None, seeds[: B * (K + 1)], pos[: B * (K + 1)], 0,
                    tok, None, d.view(-1).contiguous(), ok)
    n_acc = torch.empty(B, dtype=torch.int32, device="cuda")
    out_tok = torch.empty((B, K + 1), dtype=torch.int32, device="cuda")
    ops.accept_greedy_chain(tok.view(B, K + 1), d[:, :K].contiguous(), n_acc, out_tok)
    okm = ok.view(B, K + 1).cpu()
    for b in range(B):
        first_rej = next((j for j in range(K) if okm[b, j] == 0), K)
        assert int(n_acc[b]) == first_rej and int(out_tok[b, first_rej]) == int(tok.view(B, K + 1)[b, first_rej])


def test_speculative_sampling_with_a_stochastic_drafter(ops):
    """General speculative sampling: the drafter samples d ~ q and hands over q; the verifier accepts with
    min(1, p(d) / q(d)) and resamples from max(p - q, 0).  The emitted token must follow p, the acceptance rate must be
    sum(min(p, q))."""
    torch.manual_seed(1)
    V, n, k = 64, 8000, 8
    t_logits = (torch.randn(V) * 1.5).to(torch.bfloat16)
    d_logits = (t_logits.float() + torch.randn(V) * 1.0).to(torch.bfloat16)     # a drafter that is close, not equal
    tl = t_logits[None].repeat(n, 1).contiguous().cuda()
    dl = d_logits[None].repeat(n, 1).contiguous().cuda()
    temp = torch.ones(n, device="cuda")
    topk = torch.full((n,), k, dtype=torch.int32, device="cuda")
    seeds = torch.arange(n, dtype=torch.int64, device="cuda")
    pos = torch.full((n,), 5, dtype=torch.int32, device="cuda")
    # drafter: sample d ~ q (random stream 3) and export q
    d_tok = torch.empty(n, dtype=torch.int32, device="cuda")
    q_ids = torch.empty((n, 32), dtype=torch.int32, device="cuda")
    q_pr = torch.empty((n, 32), dtype=torch.float32, device="cuda")
    ops.sample_rows(dl, temp, topk, None, None, None, None, None, seeds, pos, 3, d_tok, None, None, None, None, None, q_ids, q_pr)
    assert bool((q_ids[:, :k] >= 0).all()) and bool((q_ids[:, k:] == -1).all())
    assert torch.allclose(q_pr.sum(1), torch.ones(n, device="cuda"), atol=1e-5)
    # verifier
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    acc = torch.empty(n, dtype=torch.int32, device="cuda")
    ops.sample_rows(tl, temp, topk, None, None, None, None, None, seeds, pos, 0, out, None, d_tok, acc, q_ids, q_pr)
    tv, ti = torch.sort(t_logits.float(), descending=True, stable=True)
    dv, di = torch.sort(d_logits.float(), descending=True, stable=True)
    p = torch.zeros(V)
    q = torch.zeros(V)
    p[ti[:k]] = torch.softmax(tv[:k], 0)
    q[di[:k]] = torch.softmax(dv[:k], 0)
    want_rate = torch.minimum(p, q).sum().item()
    assert abs(acc.float().mean().item() - want_rate) < 0.02
    emp = torch.bincount(out.cpu().long(), minlength=V).float() / n
    assert (emp - p).abs().max().item() < 0.02
    assert bool((out[acc.bool()] == d_tok[acc.bool()]).all())
    # q == p: every draft is accepted
    ops.sample_rows(tl, temp, topk, None, None, None, None, None, seeds, pos, 3, d_tok, None, None, None, None, None, q_ids, q_pr)
    ops.sample_rows(tl, temp, topk, None, None, None, None, None, seeds, pos, 0, out, None, d_tok, acc, q_ids, q_pr)
    assert acc.sum().item() == n and torch.equal(out, d_tok)


@pytest.mark.parametrize("fmt_name", ["bf16", "fp8"])
def test_selected_block_attention(ops, fmt_name):
    """Decode attention over a query-selected list of 4-token blocks plus the incomplete last block, against the
    dense oracle with the matching visibility mask; two splits of the gathered key list, scattered pages."""
    torch.manual_seed(5)
    hq, hkv, D, P = 12, 2, 256, 16
    lens = [203, 64, 1030]                        # tails of 3, 0 and 2 tokens
    B = len(lens)
    max_pages = (max(lens) + P - 1) // P
    n_pages = B * max_pages + 2
    table = torch.randperm(n_pages)[: B * max_pages].int().view(B, max_pages).cuda()
    fmt = R.KV_BF16 if fmt_name == "bf16" else R.KV_FP8_ROW
    k_codes, v_codes, k_sc, v_sc = _planes(n_pages, hkv, P, D, fmt, D)
    ks, vs = [], []
    for b, n in enumerate(lens):
        k, v = torch.randn(n, hkv, D), torch.randn(n, hkv, D)
        kq, vq = R.kv_quant_dequant(k, fmt, 64), R.kv_quant_dequant(v, fmt, 64)
        ks.append(kq); vs.append(vq)
        for t in range(n):
            page = int(table[b, t // P])
            for h in range(hkv):
                if fmt == R.KV_BF16:
                    k_codes[page, h, t % P] = k[t, h].to(torch.bfloat16).view(torch.uint8).cuda()
                    v_codes[page, h, t % P] = v[t, h].to(torch.bfloat16).view(torch.uint8).cuda()
                else:
                    for src, codes, sc in ((k[t, h], k_codes, k_sc), (v[t, h], v_codes, v_sc)):
                        x = R.bf16_round(src.float())
                        s_ = (x.abs().amax() / 448.0).clamp(2.0 ** -24, 65504.0).to(torch.float16)
                        c = (x / s_.float()).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
                        codes[page, h, t % P] = c.view(torch.uint8).cuda()
                        sc[page, h, t % P] = s_.reshape(1).view(torch.uint8).cuda()
    max_sel = 160
    sel = torch.zeros((B, max_sel), dtype=torch.int32)
    cnt = torch.zeros(B, dtype=torch.int32)
    for b, n in enumerate(lens):
        complete = n // 4
        c = min(max_sel, max(1, complete // 2))
        pick = torch.randperm(complete)[:c].sort().values if b != 1 else torch.randperm(complete)[:c]   # order is free
        sel[b, :c] = pick.int()
        cnt[b] = c
    q = torch.randn(B, hq, D).to(torch.bfloat16).cuda()
    kv_len = torch.tensor(lens, dtype=torch.int32)
    split_keys = 384
    n_splits = (4 * max_sel + 3 + split_keys - 1) // split_keys
    part_o = torch.empty(B * hq * n_splits * D, device="cuda")
    part_ml = torch.empty(B * hq * n_splits * 2, device="cuda")
    out = torch.empty((B, hq * D), dtype=torch.bfloat16, device="cuda")
    ops.paged_attention(q, hq, hkv, D, torch.arange(B).int().cuda(), kv_len.cuda(), table, k_codes, v_codes, k_sc, v_sc, P,
                        fmt, D, 1 / 16, split_keys, n_splits, part_o, part_ml, None, out, None, None, 0, False, 0,
                        sel.cuda(), cnt.cuda())
    torch.cuda.synchronize()
    for b, n in enumerate(lens):
        vis = R.selected_block_mask(kv_len[b:b + 1], sel[b:b + 1], cnt[b:b + 1], n)
        ref = R.gqa_attention(q[b:b + 1].float().cpu(), ks[b], vs[b], None, 1 / 16, vis).reshape(-1)
        err = (out[b].float().cpu() - ref).abs().max().item()
        assert err < 0.02, (fmt_name, b, err)
    with pytest.raises(RuntimeError, match="excludes a window"):
        ops.paged_attention(q, hq, hkv, D, torch.arange(B).int().cuda(), kv_len.cuda(), table, k_codes, v_codes, k_sc, v_sc,
                            P, fmt, D, 1 / 16, split_keys, n_splits, part_o, part_ml, None, out, None, None, 0, False, 128,
                            sel.cuda(), cnt.cuda())
