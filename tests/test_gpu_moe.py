"""GPU parity: MoE routing (bit-exact expert selection), permutation indices (bit-exact),
grouped GEMM + fused SwiGLU vs the CPU oracle, and batch invariance
(reference: tests/batch_invariant_ops/test_fused_moe.py:75-133, test_naive_moe.py:114-136)."""
import pytest
import torch

from conftest import load_golden
from oracle import ops

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.fixture(scope="module")
def vb():
    import vexact_b200 as vb

    vb._lib.load()
    return vb


def _seeded(*shape, seed=0, std=1.0, dtype=BF):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * std).to(dtype)


def test_route_softmax_topk_exact_indices(vb):
    for c in load_golden("route_softmax_topk"):
        w_ref, idx_ref = ops.route_softmax_topk(c["logits"], c["top_k"], True)
        w, idx = vb.route_softmax_topk(c["logits"].cuda(), c["top_k"], True)
        assert torch.equal(idx.cpu(), idx_ref)          # same tie rule as the oracle: bit-exact
        torch.testing.assert_close(w.cpu().float(), w_ref.float(), rtol=2 ** -7, atol=1e-6)
        # and against the reference's torch.topk wherever the boundary is not a tie
        probs = torch.softmax(c["logits"].float(), 1)
        srt = torch.sort(probs, descending=True).values
        distinct = (srt[:, : c["top_k"] + 1].diff(dim=1) != 0).all(dim=1)
        assert torch.equal(idx.cpu()[distinct], c["experts"][distinct])
    logits = _seeded(512, 128, seed=1, std=0.9)
    w_ref, idx_ref = ops.route_softmax_topk(logits, 8, True)
    w, idx = vb.route_softmax_topk(logits.cuda(), 8, True)
    # fp32 softmax sums may differ in the last bit between device and host; a flip needs two
    # probabilities within one fp32 ulp, so report rather than hide: require >= 99.9 % exact rows
    same = (idx.cpu() == idx_ref).all(dim=1).float().mean().item()
    assert same >= 0.999, f"expert selection differs from the oracle on {1 - same:.4%} of tokens"
    w1, idx1 = vb.route_softmax_topk(logits[:1].cuda(), 8, True)
    assert torch.equal(idx1, idx[:1]) and torch.equal(w1, w[:1])


def test_route_sigmoid_group_topk(vb):
    for c in load_golden("route_sigmoid_group_topk"):
        idx_ref, w_ref = ops.route_sigmoid_group_topk(c["logits"], c["bias"], c["n_group"], c["topk_group"],
                                                      c["top_k"], True, c["scale"])
        idx, w = vb.route_sigmoid_group_topk(c["logits"].cuda(), c["bias"].cuda(), c["n_group"], c["topk_group"],
                                             c["top_k"], True, c["scale"])
        assert torch.equal(idx.cpu(), idx_ref)
        torch.testing.assert_close(w.cpu(), w_ref, rtol=1e-5, atol=1e-6)
        assert torch.equal(torch.sort(idx.cpu(), 1).values, torch.sort(c["experts"], 1).values)


@pytest.mark.parametrize("T,k,E", [(12, 4, 8), (512, 8, 128), (2048, 8, 128), (256, 6, 64), (1, 8, 128), (3000, 2, 5),
                                   (2048, 1, 7), (2049, 1, 7), (64, 32, 200), (65, 32, 200)])
def test_moe_indices_bit_exact(vb, T, k, E):
    from vexact_b200.fused_moe import build_moe_indices

    g = torch.Generator().manual_seed(2)
    sel = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)])
    cu_ref, a_ref, sc_ref = ops.build_moe_indices(sel, E)
    cu, a_idx, sc = build_moe_indices(sel.cuda(), E)
    assert (cu.cpu().numpy() == cu_ref).all()
    assert (sc.cpu().numpy() == sc_ref).all()
    assert (a_idx.cpu().numpy() == a_ref).all()
    cu32, _, sc32 = build_moe_indices(sel.int().cuda(), E)
    assert torch.equal(cu32, cu) and torch.equal(sc32, sc)


def test_moe_indices_golden(vb):
    from vexact_b200.fused_moe import build_moe_indices

    c = load_golden("moe_indices")
    cu, a_idx, sc = build_moe_indices(c["experts"].cuda(), c["num_experts"])
    assert torch.equal(cu.cpu(), c["cu_seqlens"]) and torch.equal(a_idx.cpu(), c["a_idx"])
    assert torch.equal(sc.cpu(), c["scatter_index"])


def _moe_case(T, E, k, H, I, seed, skew=False):
    g = torch.Generator().manual_seed(seed)
    hidden = torch.randn(T, H, generator=g).to(BF)
    gate_up = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(BF)
    down = (torch.randn(E, H, I, generator=g) * 0.05).to(BF)
    if skew:
        sel = torch.stack([torch.cat([torch.zeros(1, dtype=torch.long), 1 + torch.randperm(E - 1, generator=g)[:k - 1]])
                           for _ in range(T)])
    else:
        sel = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)])
    rw = torch.rand(T, k, generator=g)
    rw = (rw / rw.sum(-1, keepdim=True)).to(BF)
    return hidden, gate_up, down, sel, rw


@pytest.mark.parametrize("T,E,k,H,I,skew", [(12, 8, 4, 64, 32, False), (64, 16, 4, 256, 128, False),
                                            (300, 8, 2, 512, 192, True), (40, 128, 8, 2048, 768, False)])
def test_fused_moe_oracle(vb, T, E, k, H, I, skew):
    hidden, gate_up, down, sel, rw = _moe_case(T, E, k, H, I, seed=3, skew=skew)
    ref = ops.fused_moe_batched(E, rw, sel, hidden, gate_up[:, :I], gate_up[:, I:], down)
    out = vb.fused_moe_forward(E, rw.cuda(), sel.cuda(), hidden.cuda(), fc2_weight=down.cuda(),
                               fc1_1_2_weight=gate_up.cuda())
    # Each of the k expert rows summed into a token is a bf16 tensor, and a one-ulp flip of an
    # intermediate (device expf / accumulation order) moves a row by one bf16 ulp of the ROW's
    # magnitude, which can exceed an ulp of a sum that cancels.  Stated tolerance: 2^-6 of the
    # largest output magnitude, absolute; and at least 95 % of elements bit-identical.
    tol = 2 ** -6 * max(ref.float().abs().max().item(), 1e-3)
    torch.testing.assert_close(out.cpu().float(), ref.float(), rtol=0, atol=tol)
    assert (out.cpu() == ref).float().mean() > 0.95
    # split gate / up weights (the reference's positional signature) give the same bits
    out_split = vb.fused_moe_forward(E, rw.cuda(), sel.cuda(), hidden.cuda(), gate_up[:, :I].contiguous().cuda(),
                                     gate_up[:, I:].contiguous().cuda(), down.cuda())
    assert torch.equal(out_split, out)


def test_fused_moe_golden_naive(vb):
    c = load_golden("moe_naive")
    E = c["gate_up"].shape[0]
    out = vb.fused_moe_forward(E, c["weights"].cuda(), c["experts"].cuda(), c["hidden"].cuda(),
                               fc2_weight=c["down"].cuda(), fc1_1_2_weight=c["gate_up"].cuda())
    err = (out.cpu().float() - c["out_fp32"]).abs().max().item()
    assert err < 2e-3 * max(1.0, c["out_fp32"].abs().max().item())


def test_fused_moe_batch_invariance_bitwise(vb):
    """Full batch vs token by token: identical bits (the reference allows 1e-3 here)."""
    T, E, k, H, I = 96, 32, 4, 512, 256
    hidden, gate_up, down, sel, rw = _moe_case(T, E, k, H, I, seed=4)
    args = (down.cuda(), gate_up.cuda())
    full = vb.fused_moe_forward(E, rw.cuda(), sel.cuda(), hidden.cuda(), fc2_weight=args[0], fc1_1_2_weight=args[1])
    for t in (0, 1, 17, 95):
        one = vb.fused_moe_forward(E, rw[t:t + 1].cuda(), sel[t:t + 1].cuda(), hidden[t:t + 1].cuda(),
                                   fc2_weight=args[0], fc1_1_2_weight=args[1])
        assert torch.equal(one, full[t:t + 1]), f"token {t} differs between batch {T} and batch 1"
    half = vb.fused_moe_forward(E, rw[:40].cuda(), sel[:40].cuda(), hidden[:40].cuda(), fc2_weight=args[0],
                                fc1_1_2_weight=args[1])
    assert torch.equal(half, full[:40])


def test_status_word_clean(vb):
    torch.cuda.synchronize()
    assert vb._lib.read_status()[0] == 0


def test_deferred_topk_sum_fused_with_add_rmsnorm_bitwise(vb):
    """PendingMoE.add_norm == finish() followed by add_rms_norm, bit for bit (with and without addend)."""
    for H in (2048, 512):      # one-CTA-per-row norm (fused kernel) and the short-row fallback
        _check_deferred_sum(vb, H)


def _check_deferred_sum(vb, H):
    g = torch.Generator().manual_seed(5)
    T, E, k, I = 96, 16, 4, 256
    x = (torch.randn(T, H, generator=g) * 0.5).bfloat16().cuda()
    w13 = (torch.randn(E, 2 * I, H, generator=g) * 0.05).bfloat16().cuda()
    w2 = (torch.randn(E, H, I, generator=g) * 0.05).bfloat16().cuda()
    logits = torch.randn(T, E, generator=g).bfloat16().cuda()
    rw, sel = vb.route_softmax_topk(logits, k, True)
    residual = torch.randn(T, H, generator=g).bfloat16().cuda()
    norm_w = (1 + 0.02 * torch.randn(H, generator=g)).bfloat16().cuda()
    for addend in (None, (torch.randn(T, H, generator=g) * 0.3).bfloat16().cuda()):
        for hf in (True, False):
            plain = vb.fused_moe_forward(E, rw, sel, x, fc2_weight=w2, fc1_1_2_weight=w13, addend=addend)
            want_sum, want_norm = vb.add_rms_norm(plain, residual, norm_w, 1e-6, hf=hf)
            pend = vb.fused_moe_forward(E, rw, sel, x, fc2_weight=w2, fc1_1_2_weight=w13, addend=addend,
                                        defer_reduce=True)
            got_sum, got_norm = pend.add_norm(residual, norm_w, 1e-6, hf=hf)
            assert torch.equal(got_sum, want_sum) and torch.equal(got_norm, want_norm)
            assert torch.equal(pend.finish(), plain)


def test_fc1_routes_agree_bitwise(vb):
    """fc1 with the fused SwiGLU epilogue (few rows per expert) and as plain grouped GEMM + elementwise
    kernel (many rows per expert): the same token gets the same bits."""
    g = torch.Generator().manual_seed(31)
    T, E, k, H, I = 600, 8, 2, 256, 128          # 150 rows per expert: split route
    x = (torch.randn(T, H, generator=g) * 0.5).bfloat16().cuda()
    w13 = (torch.randn(E, 2 * I, H, generator=g) * 0.05).bfloat16().cuda()
    w2 = (torch.randn(E, H, I, generator=g) * 0.05).bfloat16().cuda()
    logits = torch.randn(T, E, generator=g).bfloat16().cuda()
    rw, sel = vb.route_softmax_topk(logits, k, True)
    big = vb.fused_moe_forward(E, rw, sel, x, fc2_weight=w2, fc1_1_2_weight=w13)
    small = vb.fused_moe_forward(E, rw[:100], sel[:100], x[:100], fc2_weight=w2, fc1_1_2_weight=w13)   # 25 per expert: fused
    assert torch.equal(big[:100], small)


@pytest.mark.parametrize("T,E,k,H,I,skew", [(1, 8, 2, 64, 32, False), (7, 16, 4, 256, 128, False),
                                            (300, 8, 2, 512, 192, True), (512, 128, 8, 2048, 768, False),
                                            (600, 8, 2, 256, 128, False)])
def test_fc1_gathering_its_rows_equals_the_permuted_copy_bitwise(vb, monkeypatch, T, E, k, H, I, skew):
    """fc1 reading x[gather_index[r]] (one-row TMA boxes, four rows per gather) against fc1 over the
    expert-sorted copy of x: the same bytes land in the same shared-memory rows, so every output bit agrees;
    with fused and with split fc1 weights, and from a strided view of the activations."""
    hidden, gate_up, down, sel, rw = _moe_case(T, E, k, H, I, seed=11, skew=skew)
    args = (E, rw.cuda(), sel.cuda())
    wide = torch.zeros(T, H + 64, dtype=BF, device="cuda")
    wide[:, :H] = hidden.cuda()
    outs = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("B200_MOE_GATHER", mode)
        outs[mode] = (
            vb.fused_moe_forward(*args, hidden.cuda(), fc2_weight=down.cuda(), fc1_1_2_weight=gate_up.cuda()),
            vb.fused_moe_forward(*args, hidden.cuda(), gate_up[:, :I].contiguous().cuda(),
                                 gate_up[:, I:].contiguous().cuda(), down.cuda()),
            vb.fused_moe_forward(*args, wide[:, :H], fc2_weight=down.cuda(), fc1_1_2_weight=gate_up.cuda()),
        )
    for a, b in zip(outs["0"], outs["1"]):
        assert torch.equal(a, b)
    assert torch.equal(outs["1"][0], outs["1"][2])


@pytest.mark.parametrize("T,E,k,H,I,skew", [(1, 8, 2, 64, 32, False), (40, 128, 8, 2048, 768, False),
                                            (512, 128, 8, 2048, 768, False), (300, 8, 2, 512, 192, True)])
def test_routing_with_its_plan_equals_route_index_scatter_bitwise(vb, T, E, k, H, I, skew):
    """Routing that hands out the permutation itself (two launches) against route -> index -> scatter (three):
    same routing weights and experts, cu_seqlens and tile table; the rows of an expert's group may sit in another
    order, and every output of the MoE is the same bits.  Twice in a row: the counters come back clean."""
    from vexact_b200.fused_moe import _PLAN_COUNTERS, _permute, route_plan_softmax_topk

    hidden, gate_up, down, _, _ = _moe_case(T, E, k, H, I, seed=21, skew=skew)
    g = torch.Generator().manual_seed(4)
    logits = (torch.randn(T, E, generator=g) * (3.0 if skew else 1.0)).to(BF).cuda()
    x, gu, dn = hidden.cuda(), gate_up.cuda(), down.cuda()
    rw0, sel0 = vb.route_softmax_topk(logits, k, True)
    want = vb.fused_moe_forward(E, rw0, sel0, x, fc2_weight=dn, fc1_1_2_weight=gu)
    classic = _permute(sel0, rw0, None, E)
    for _ in range(2):
        rw, sel, plan = route_plan_softmax_topk(logits, k, True, E)
        assert torch.equal(rw, rw0) and torch.equal(sel, sel0)
        assert torch.equal(plan["cu_seqlens"], classic["cu_seqlens"])
        assert torch.equal(plan["tile_count"], classic["tile_count"])
        nt = int(plan["tile_count"])
        assert torch.equal(plan["tile_table"][:nt], classic["tile_table"][:nt])
        # ranks: within every expert exactly 0 .. count-1
        cnt = torch.bincount(sel.flatten(), minlength=E)
        for e in range(E):
            r = plan["rank"][(sel.flatten() == e)].sort().values
            assert torch.equal(r, torch.arange(int(cnt[e]), device="cuda", dtype=torch.int32))
        got = vb.fused_moe_forward(E, rw, sel, x, fc2_weight=dn, fc1_1_2_weight=gu, plan=plan)
        assert torch.equal(got, want)
        torch.cuda.synchronize()
        assert int(_PLAN_COUNTERS[torch.cuda.current_device()].abs().sum()) == 0


def test_gather_index_is_the_inverse_of_scatter_index(vb):
    from vexact_b200.fused_moe import _permute

    g = torch.Generator().manual_seed(5)
    T, k, E = 333, 6, 64
    sel = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)]).cuda()
    rw = torch.rand(T, k, generator=g).bfloat16().cuda()
    plan = _permute(sel, rw, None, E, gather=True)
    scatter = plan["scatter_index"].long()
    n = T * k
    assert torch.equal(scatter.sort().values, torch.arange(n, device="cuda"))
    want = torch.empty(n, dtype=torch.int32, device="cuda")
    want[scatter] = (torch.arange(n, device="cuda") // k).int()
    assert torch.equal(plan["gather_index"], want)
    scale = torch.empty(n, dtype=BF, device="cuda")
    scale[scatter] = rw.flatten()
    assert torch.equal(plan["row_scale"], scale)
    # within an expert the rows keep token order (stable sort), as the reference's argsort(stable=True) gives
    cu = plan["cu_seqlens"].tolist()
    gi = plan["gather_index"].tolist()
    assert all(gi[a:b] == sorted(gi[a:b]) for a, b in zip(cu[:-1], cu[1:]))


@pytest.mark.gpu
def test_routing_of_nan_rows_stays_in_range():
    """Padded tokens of a captured batch carry undefined (possibly NaN) hidden states; their routing must
    still name experts inside [0, E) so that nothing downstream indexes out of range."""
    import vexact_b200 as vb

    E, k = 64, 6
    logits = torch.randn(5, E, device="cuda")
    logits[1] = float("nan")
    logits[3, 7] = float("nan")
    _, sel = vb.route_softmax_topk(logits, k, True)
    assert int(sel.min()) >= 0 and int(sel.max()) < E
    idx, _ = vb.route_sigmoid_group_topk(logits, torch.zeros(E, device="cuda"), 4, 2, k, True, 2.5)
    assert int(idx.min()) >= 0 and int(idx.max()) < E
    # rows without NaN are untouched by the guard
    clean = logits[[0, 2, 4]].contiguous()
    _, sel_c = vb.route_softmax_topk(clean, k, True)
    assert torch.equal(sel_c, sel[[0, 2, 4]])
    torch.cuda.synchronize()
    assert vb._lib.read_status()[0] == 0


def test_group_gemm_operators_under_the_reference_names(vb):
    """`expert_histogram`, `moe_scatter`, `group_gemm_same_nk`, `moe_gather` (reference group_gemm/kernel/moe.py:52,
    :304, :131; group_gemm.py:156) one at a time, chained as FusedMoeExpertFunction.forward chains them
    (fused_moe.py:24-111): index and copy steps bit-exact, the GEMM equal to the dense GEMM's bits per expert,
    the chain equal to `fused_moe_forward` up to the activation's rounding."""
    from vexact_b200 import group_gemm as gg

    T, E, k, H, I = 70, 16, 4, 256, 128
    hidden, gate_up, down, sel, rw = _moe_case(T, E, k, H, I, seed=11)
    x, sel_d, rw_d = hidden.cuda(), sel.cuda(), rw.cuda()
    w1, w2, w3 = gate_up[:, :I].contiguous().cuda(), gate_up[:, I:].contiguous().cuda(), down.cuda()

    splits = gg.expert_histogram(sel_d, E)
    assert splits.dtype == torch.int32
    assert torch.equal(splits.cpu().long(), torch.bincount(sel.flatten(), minlength=E))
    assert torch.equal(gg.expert_histogram(sel_d.int(), E), splits)

    scatter_index = sel_d.flatten().argsort(stable=True).argsort().int().view(sel_d.shape)   # fused_moe.py:43
    cu, a_idx, scatter_ours = vb.fused_moe.build_moe_indices(sel_d, E)
    assert torch.equal(scatter_ours, scatter_index)

    rows = gg.moe_index_compute(sel_d, torch.cumsum(splits, dim=0))     # moe.py:382: any order inside an expert;
    assert rows.dtype == torch.int64 and torch.equal(rows, scatter_index.long())   # here the stable one

    scattered = gg.moe_scatter(x, scatter_index)
    assert torch.equal(scattered, x[a_idx.long()])
    assert torch.equal(gg.moe_scatter(x.half(), scatter_index.long()), x.half()[a_idx.long()])   # fp16 rows, int64 index

    cumsum_t = torch.cumsum(splits, dim=0)
    fc1_1 = gg.group_gemm_same_nk(a=scattered, b=w1, cumsum_M=cumsum_t, max_M=scattered.shape[0], transpose_b=True)
    fc1_2 = gg.group_gemm_same_nk(a=scattered, b=w2, cumsum_M=cumsum_t, max_M=scattered.shape[0], transpose_b=True)
    bounds = [0] + cumsum_t.tolist()
    for e in range(E):          # a token's dot products do not depend on the tile it sits in: the dense GEMM's bits
        lo, hi = bounds[e], bounds[e + 1]
        if hi > lo:
            assert torch.equal(fc1_1[lo:hi], vb.matmul_persistent(scattered[lo:hi], w1[e].t()))
    ref32 = torch.cat([scattered[bounds[e]:bounds[e + 1]].float() @ w2[e].float().t() for e in range(E)])
    torch.testing.assert_close(fc1_2.float(), ref32, rtol=2 ** -7, atol=2 ** -7 * ref32.abs().max().item())

    gate_w = torch.empty(T * k, 1, dtype=BF, device="cuda")
    gate_w[scatter_index.flatten().long()] = rw_d.reshape(-1, 1)                               # fused_moe.py:84-86
    weighted = torch.ops.aten.silu(fc1_1) * fc1_2 * gate_w
    fc2 = gg.group_gemm_same_nk(a=weighted, b=w3, cumsum_M=cumsum_t, max_M=weighted.shape[0], transpose_b=True)

    out = gg.moe_gather(fc2, scatter_index)
    acc = torch.zeros(T, H, device="cuda")
    for j in range(k):                                   # fp32 sum in k order, one rounding (moe.py:113-127)
        acc += fc2[scatter_index[:, j].long()].float()
    assert torch.equal(out, acc.to(BF))

    fused = vb.fused_moe_forward(E, rw_d, sel_d, x, w1, w2, w3)
    tol = 2 ** -6 * max(fused.float().abs().max().item(), 1e-3)
    torch.testing.assert_close(out.float(), fused.float(), rtol=0, atol=tol)
    assert (out == fused).float().mean() > 0.95

    # the two GEMM forms of the backward (group_gemm.py:156 with transpose_b=False, :360 group_gemm_same_mn)
    dgrad = gg.group_gemm_same_nk(fc1_1, w1, cumsum_t, T * k, transpose_b=False)        # [R, I] x [E, I, H] -> [R, H]
    assert torch.equal(dgrad, gg.group_gemm_same_nk(fc1_1, w1.transpose(1, 2).contiguous(), cumsum_t, T * k,
                                                    transpose_b=True))
    ref32 = torch.cat([fc1_1[bounds[e]:bounds[e + 1]].float() @ w1[e].float() for e in range(E)])
    torch.testing.assert_close(dgrad.float(), ref32, rtol=2 ** -7, atol=2 ** -7 * ref32.abs().max().item())
    wgrad = gg.group_gemm_same_mn(fc1_1, scattered, torch.full_like(w1, 7.0), cumsum_t, T * k, transpose_a=True,
                                  transpose_b=False)                                  # [E, I, H]
    ref32 = torch.stack([fc1_1[bounds[e]:bounds[e + 1]].float().t() @ scattered[bounds[e]:bounds[e + 1]].float()
                         for e in range(E)])
    torch.testing.assert_close(wgrad.float(), ref32, rtol=2 ** -7, atol=2 ** -8 * ref32.abs().max().item())
    lonely = torch.cumsum(torch.tensor([3, 0, T * k - 3] + [0] * (E - 3), device="cuda"), 0)   # empty groups: zeros
    wz = gg.group_gemm_same_mn(fc1_1, scattered, torch.full_like(w1, 7.0), lonely, T * k, transpose_a=True,
                               transpose_b=False)
    assert not wz[1].any() and not wz[3:].any() and wz[0].any() and wz[2].any()
    torch.cuda.synchronize()
    assert vb._lib.read_status()[0] == 0
    overrun = lonely.clone()
    overrun[-1] = T * k + 9                                  # past the last row: clipped and reported
    wo = gg.group_gemm_same_mn(fc1_1, scattered, torch.full_like(w1, 7.0), overrun, T * k, transpose_a=True,
                               transpose_b=False)
    torch.cuda.synchronize()
    assert vb._lib.read_status()[:2] == (2, E - 1)
    assert torch.equal(wo[2], wz[2]) and not wo[E - 1].any()

    for call in (lambda: gg.group_gemm_same_mn(scattered, scattered, w1, cumsum_t, T * k),
                 lambda: gg.moe_add_gather(fc2, fc2, scatter_index)):
        with pytest.raises(NotImplementedError):
            call()


def test_scatter_and_gather_skip_and_report_an_index_out_of_range(vb):
    from vexact_b200 import group_gemm as gg

    T, k, H = 6, 2, 64
    x = _seeded(T, H, seed=2).cuda()
    index = torch.randperm(T * k, generator=torch.Generator().manual_seed(3)).int().view(T, k).cuda()
    good = gg.moe_scatter(x, index)
    torch.cuda.synchronize()
    assert vb._lib.read_status()[0] == 0
    bad = index.clone()
    bad[4, 1] = T * k + 5
    gg.moe_scatter(x, bad)
    torch.cuda.synchronize()
    code, detail, _, _ = vb._lib.read_status()
    assert (code, detail) == (2, 4 * k + 1)
    rows = _seeded(T * k, H, seed=4).cuda()
    bad[4, 1] = -3
    out = gg.moe_gather(rows, bad)
    torch.cuda.synchronize()
    code, detail, _, _ = vb._lib.read_status()
    assert (code, detail) == (2, 4 * k + 1)
    assert torch.equal(out[4], rows[bad[4, 0].long()])          # the bad term contributes nothing
    assert torch.equal(out[:4], gg.moe_gather(rows, index)[:4])
    assert vb._lib.read_status()[0] == 0
    assert good.shape == (T * k, H)


def test_expert_function_classes_take_the_reference_arguments(vb):
    """`FusedMoeExpertFunction.apply` / `QuackFusedMoeExpertFunction.apply` (fused_moe.py:22, :295) with the
    reference's seven positional arguments: the fused forward's bits."""
    from vexact_b200.fused_moe import FusedMoeExpertFunction, QuackFusedMoeExpertFunction

    T, E, k, H, I = 33, 8, 2, 128, 64
    hidden, gate_up, down, sel, rw = _moe_case(T, E, k, H, I, seed=21)
    args = (E, rw.cuda(), sel.cuda(), hidden.cuda(), gate_up[:, :I].contiguous().cuda(),
            gate_up[:, I:].contiguous().cuda(), down.cuda())
    fused = vb.fused_moe_forward(*args)
    assert torch.equal(FusedMoeExpertFunction.apply(*args), fused)
    assert torch.equal(QuackFusedMoeExpertFunction.apply(*args), fused)


@pytest.mark.parametrize("fused_weights", [False, True])
def test_fused_moe_backward_against_autograd_of_the_fp32_formula(vb, fused_weights):
    """Gradients of `fused_moe_forward` (reference backward: fused_moe.py:113-265) for the hidden states, the routing
    weights and the three weight tensors, against torch autograd on the fp32 statement of the same function
    (sum over k of w_k * fc2_e(silu(fc1_1_e x) * fc1_2_e x)).  The chain rounds to bf16 after every step, as the
    reference's does: stated tolerance 2^-5 of each gradient's largest magnitude, and cosine similarity > 0.999.
    One expert is never selected: its weight gradients are exact zeros."""
    T, E, k, H, I = 48, 8, 2, 128, 64
    hidden, gate_up, down, sel, rw = _moe_case(T, E, k, H, I, seed=31)
    sel = torch.where(sel == E - 1, torch.zeros_like(sel), sel)          # expert E-1 unused
    dup = sel[:, 0] == sel[:, 1]
    sel[dup, 1] = (sel[dup, 0] + 1) % (E - 1)
    g_out = _seeded(T, H, seed=32)
    leaves = dict(x=hidden.cuda(), rw=rw.cuda(), w1=gate_up[:, :I].contiguous().cuda(),
                  w2=gate_up[:, I:].contiguous().cuda(), w3=down.cuda())
    ours = {n: t.clone().requires_grad_(True) for n, t in leaves.items()}
    if fused_weights:       # the model files' keyword form: one [E, 2I, H] tensor, gate rows first
        gu = torch.cat([ours["w1"], ours["w2"]], dim=1)
        out = vb.fused_moe_forward(E, ours["rw"], sel.cuda(), ours["x"], fc2_weight=ours["w3"], fc1_1_2_weight=gu)
    else:
        out = vb.fused_moe_forward(E, ours["rw"], sel.cuda(), ours["x"], ours["w1"], ours["w2"], ours["w3"])
    assert torch.equal(out, vb.fused_moe_forward(E, leaves["rw"], sel.cuda(), leaves["x"], leaves["w1"], leaves["w2"],
                                                 leaves["w3"]))
    out.backward(g_out.cuda())

    ref = {n: t.float().clone().requires_grad_(True) for n, t in leaves.items()}
    s = sel.cuda()
    acc = torch.zeros(T, H, device="cuda")
    for j in range(k):
        e = s[:, j]
        a = torch.einsum("th,tih->ti", ref["x"], ref["w1"][e])
        b = torch.einsum("th,tih->ti", ref["x"], ref["w2"][e])
        acc = acc + torch.einsum("ti,thi->th", torch.nn.functional.silu(a) * b * ref["rw"][:, j:j + 1], ref["w3"][e])
    acc.backward(g_out.cuda().float())
    for n in leaves:
        got, want = ours[n].grad.float(), ref[n].grad
        assert got.shape == want.shape and ours[n].grad.dtype == leaves[n].dtype
        tol = 2 ** -5 * want.abs().max().item()
        torch.testing.assert_close(got, want, rtol=0, atol=tol, msg=lambda m, n=n: f"grad of {n}: {m}")
        cos = torch.nn.functional.cosine_similarity(got.flatten(), want.flatten(), dim=0).item()
        assert cos > 0.999, (n, cos)
    for n in ("w1", "w2", "w3"):
        assert not ours[n].grad[E - 1].any()


@pytest.mark.parametrize("stacked", [False, True])
@pytest.mark.parametrize("T, E, k, H, I", [(64, 16, 4, 512, 256), (150, 8, 2, 512, 200), (1100, 6, 2, 256, 128)])
def test_fused_moe_backward_rounds_as_the_chain_of_operators(vb, T, E, k, H, I, stacked):
    """The backward against the reference's chain (fused_moe.py:113-236) of single operators under its names and torch's
    silu_backward: the same bits for every gradient, whatever the width (multiples of 64 or not) and the storage of fc1's
    weights.  The routing weights' gradient is an fp32 sum of I bf16 values in another order, so one bf16 rounding apart."""
    from vexact_b200 import group_gemm as gg

    hidden, gate_up, down, sel, rw = (t.cuda() for t in _moe_case(T, E, k, H, I, seed=77))
    gate_up, g_out = gate_up * 4, _seeded(T, H, seed=78).cuda()         # gates spread over the bend of silu
    x, w3, wr = (t.clone().requires_grad_() for t in (hidden, down, rw))
    if stacked:
        leaves = [gate_up.clone().requires_grad_()]
        out = vb.fused_moe_forward(E, wr, sel, x, fc2_weight=w3, fc1_1_2_weight=leaves[0])
    else:
        leaves = [gate_up[:, i * I:(i + 1) * I].clone().requires_grad_() for i in (0, 1)]
        out = vb.fused_moe_forward(E, wr, sel, x, *leaves, w3)
    got = torch.autograd.grad(out, [wr, x, w3, *leaves], g_out)

    w1, w2 = gate_up[:, :I].contiguous(), gate_up[:, I:].contiguous()
    cu, _, index = vb.fused_moe.build_moe_indices(sel, E)
    ends, rows, at = cu[1:], T * k, index.flatten().long()

    def product(a, w, forward):
        return gg.group_gemm_same_nk(a, w, ends, rows, transpose_b=forward)

    def weight(a, b, like):
        return gg.group_gemm_same_mn(a, b, torch.empty_like(like), ends, rows, transpose_a=True, transpose_b=False)

    xs, g_y = gg.moe_scatter(hidden, index), gg.moe_scatter(g_out, index)
    gate, up = product(xs, w1, True), product(xs, w2, True)
    act = torch.nn.functional.silu(gate) * up
    row_w = torch.empty((rows, 1), dtype=BF, device="cuda")
    row_w[at] = rw.reshape(-1, 1)
    g_in = product(g_y, down, False)
    g_act = g_in * row_w
    g_up, g_gate = torch.nn.functional.silu(gate) * g_act, torch.ops.aten.silu_backward(g_act * up, gate)
    g_xs = product(g_gate, w1, False) + product(g_up, w2, False)
    torch.testing.assert_close(got[0], (act * g_in).sum(-1)[at].reshape(rw.shape), rtol=2 ** -7, atol=1e-6 * I)
    assert torch.equal(got[1], gg.moe_gather(g_xs, index))
    assert torch.equal(got[2], weight(g_y, act * row_w, down))
    assert torch.equal(torch.cat(got[3:], 1), torch.cat([weight(g_gate, xs, w1), weight(g_up, xs, w2)], 1))


def test_weight_gradient_kernels_tensor_core_and_cuda_core_forms(vb):
    """`group_gemm_same_mn` runs on the tensor cores when M and N are multiples of 8 and on the CUDA cores
    otherwise; both against the fp32 product, with ragged and empty groups and tiles that overhang M and N."""
    from vexact_b200 import group_gemm as gg

    g = torch.Generator().manual_seed(41)
    counts = [0, 37, 1, 200, 0, 16, 90]
    R, G = sum(counts), len(counts)
    cs = torch.cumsum(torch.tensor(counts), 0).cuda()
    bounds = [0] + cs.tolist()
    for M, N in [(200, 136), (128, 256), (36, 20)]:
        a = torch.randn(R, M, generator=g).to(BF).cuda()
        b = torch.randn(R, N, generator=g).to(BF).cuda()
        c = gg.group_gemm_same_mn(a, b, torch.full((G, M, N), 7.0, dtype=BF, device="cuda"), cs, R, transpose_a=True,
                                  transpose_b=False)
        ref = torch.stack([a[bounds[e]:bounds[e + 1]].float().t() @ b[bounds[e]:bounds[e + 1]].float() for e in range(G)])
        torch.testing.assert_close(c.float(), ref, rtol=2 ** -7, atol=2 ** -8 * ref.abs().max().item())
        assert not c[0].any() and not c[4].any()
    torch.cuda.synchronize()
    assert vb._lib.read_status()[0] == 0


@pytest.mark.parametrize("E,k,T,H,I", [(4, 2, 150, 256, 200), (3, 1, 1111, 128, 72), (8, 4, 260, 192, 328)])
def test_grouped_gemm_tile_heights_and_unfused_swiglu(vb, E, k, T, H, I):
    """More than 64 rows per expert: tiles of up to 128 or 256 rows, cut evenly in steps of 16 and fetched in boxes by the
    binary digits of their height.  A row's bits do not depend on its tile, so every tile height gives those of 64-row tiles;
    the elementwise SwiGLU (16 bytes per thread, or 2 where a row stride does not allow it) rounds as the fused epilogue."""
    from vexact_b200 import _lib, fused_moe as fm

    g = torch.Generator().manual_seed(E * T)
    x = torch.randn(T, H, generator=g).to(BF).cuda()
    w = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(BF).cuda()
    sel = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)]).cuda()
    sel[: T // 2, 0] = sel[0, 0]                       # one crowded expert (top-1 or not: duplicates are rows of their own)
    rw = torch.rand(T, k, generator=g).to(BF).cuda()
    assert T * k > 64 * E
    plan = fm._permute(sel, rw, x, E)
    count = int(plan["tile_count"])
    table = plan["tile_table"][:count].cpu()
    cu = plan["cu_seqlens"].cpu()
    for e in range(E):                                 # the tiles of an expert cover its rows, in order, evenly
        mine = table[table[:, 0] == e]
        rows = int(cu[e + 1] - cu[e])
        assert mine[:, 2].sum() == rows and len(mine) == -(-rows // plan["tile_rows"])
        if rows:
            assert mine[0, 1] == cu[e] and mine[:, 2].max() <= plan["tile_rows"] and mine[:, 2].min() > 0
            assert torch.equal(mine[1:, 1], mine[:-1, 1] + mine[:-1, 2])
    tall = fm._grouped_gemm(plan["x_perm"], w, None, plan, 2 * I, mode=0)
    low = dict(plan, tile_rows=64)
    rows64 = [(e, r, min(64, int(cu[e + 1]) - r), 0) for e in range(E) for r in range(int(cu[e]), int(cu[e + 1]), 64)]
    low.update(tile_table=torch.tensor(rows64, dtype=torch.int32).cuda(), max_tiles=len(rows64),
               tile_count=torch.tensor([len(rows64)], dtype=torch.int32).cuda())
    assert torch.equal(tall, fm._grouped_gemm(plan["x_perm"], w, None, low, 2 * I, mode=0))
    fused = fm._grouped_gemm(plan["x_perm"], w, plan["row_scale"], low, I, mode=1)
    odd = torch.empty(tall.shape[0], 2 * I + 2, dtype=BF, device="cuda")          # a row stride without 16-byte rows
    odd[:, :2 * I] = tall
    for gu in (tall, odd):
        h = torch.empty_like(fused)
        _lib.check(_lib.load().b200_swiglu_scale_strided(gu.data_ptr(), gu.data_ptr() + 2 * I, plan["row_scale"].data_ptr(),
                                                         h.data_ptr(), gu.shape[0], I, gu.stride(0), _lib.current_stream()), "swiglu")
        assert torch.equal(h, fused)
    torch.cuda.synchronize()
    assert vb._lib.read_status()[0] == 0


def _tile_table(cu, height):
    rows = [(e, r, min(height, cu[e + 1] - r), 0) for e in range(len(cu) - 1) for r in range(cu[e], cu[e + 1], height)]
    return dict(tile_table=torch.tensor(rows, dtype=torch.int32, device="cuda"), max_tiles=len(rows), tile_rows=height,
                tile_count=torch.tensor([len(rows)], dtype=torch.int32, device="cuda"))


@pytest.mark.parametrize("K", [192, 200])
@pytest.mark.parametrize("height", [16, 48, 80, 96, 112, 144, 176, 208, 240, 256])
def test_grouped_products_at_every_tile_height(vb, height, K):
    """Every multiple of 16 up to 256 is a tile height, also those above 64 that are no multiple of the 32 columns in which CTA
    pairs take tiles: the bits of 64-row tiles, for the plain, gated, squared and data-gradient products, with full tiles
    and more of them than the pairs of the chip.  The sum of two data gradients is that of the rounded two."""
    from vexact_b200 import _lib, fused_moe as fm

    E, N, cu = 3, 2048, [0, 700, 1411, 2111]
    gen = torch.Generator(device="cuda").manual_seed(height + K)
    R = cu[-1]
    x = torch.randn(R, K, device="cuda", generator=gen).to(BF)
    w = (torch.randn(E, N, K, device="cuda", generator=gen) * 0.1).to(BF)
    wt, x2 = w.transpose(1, 2).contiguous(), torch.randn(R, K, device="cuda", generator=gen).to(BF)
    wt2 = (torch.randn(E, K, N, device="cuda", generator=gen) * 0.1).to(BF)
    scale = torch.rand(R, device="cuda", generator=gen).to(BF)

    def products(plan):
        common = plan["tile_table"].data_ptr(), plan["tile_count"].data_ptr()
        act, back, other, both = (torch.empty(R, N, dtype=BF, device="cuda") for _ in range(4))
        _lib.check(_lib.load().b200_moe_grouped_gemm_act(
            x.data_ptr(), w.data_ptr(), None, act.data_ptr(), *common, R, E, N, K, N, plan["max_tiles"], plan["tile_rows"], 3,
            _lib.current_stream()), "act")
        for rows, weights, out in ((x, wt, back), (x2, wt2, other)):
            _lib.check(_lib.load().b200_moe_grouped_dgrad(
                rows.data_ptr(), weights.data_ptr(), None, out.data_ptr(), *common, R, E, N, K, N, plan["max_tiles"],
                plan["tile_rows"], _lib.current_stream()), "dgrad")
        pair, stacked = torch.cat([x, x2], 1), torch.cat([wt, wt2], 1)      # both halves as they lie in one tensor
        _lib.check(_lib.load().b200_moe_grouped_dgrad_sum(
            pair.data_ptr(), pair[:, K:].data_ptr(), 2 * K, stacked.data_ptr(), stacked[:, K:].data_ptr(), 2 * K * N, both.data_ptr(),
            *common, R, E, N, K, N, plan["max_tiles"], plan["tile_rows"], _lib.current_stream()), "dgrad_sum")
        assert torch.equal(both, back + other)
        return (fm._grouped_gemm(x, w, None, plan, N, mode=0), fm._grouped_gemm(x, w, scale, plan, N // 2, mode=1), act, back)

    for got, want in zip(products(_tile_table(cu, height)), products(_tile_table(cu, 64))):
        assert torch.equal(got, want)
    torch.cuda.synchronize()
    assert vb._lib.read_status()[0] == 0


@pytest.mark.parametrize("tile_rows", [1, 7, 16, 24, 40, 64, 100, 200, 256])
def test_tile_tables_cover_the_rows_at_any_height(vb, tile_rows):
    """A token tile has at least one row and at most tile_rows, whatever tile_rows is, and an expert's tiles cover its rows in
    order, as few as they can be."""
    from vexact_b200 import _lib

    counts = [0, 1, 15, 16, 17, 201, 40, 333, 0, 64, 640]
    E, n = len(counts), sum(counts)
    sel = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))
    sel = sel[torch.randperm(n, generator=torch.Generator().manual_seed(tile_rows))].cuda()
    max_tiles = sum(-(-c // tile_rows) for c in counts)
    index, cu, table, count, gather = (torch.zeros(s, dtype=torch.int32, device="cuda") for s in (n, E + 1, (max_tiles, 4), 1, n))
    _lib.check(_lib.load().b200_moe_permute_index(
        sel.data_ptr(), 1, None, index.data_ptr(), cu.data_ptr(), gather.data_ptr(), None, table.data_ptr(), count.data_ptr(), n, 1,
        E, tile_rows, max_tiles, _lib.current_stream()), "permute")
    _check_tiles(table[:int(count)].tolist(), counts, tile_rows)
    T = 150
    logits = torch.randn(T, E, generator=torch.Generator().manual_seed(5)).cuda()
    logits[:, 3] += 3.0
    weights, rank = torch.empty(T, 2, dtype=BF, device="cuda"), torch.empty(2 * T, dtype=torch.int32, device="cuda")
    chosen = torch.empty(T, 2, dtype=torch.int64, device="cuda")
    counters = torch.zeros(1024, dtype=torch.int32, device="cuda")
    table = torch.zeros(2 * T + E, 4, dtype=torch.int32, device="cuda")
    _lib.check(_lib.load().b200_moe_route_plan_softmax_topk(
        logits.data_ptr(), 0, E, weights.data_ptr(), chosen.data_ptr(), rank.data_ptr(), counters.data_ptr(), cu.data_ptr(),
        table.data_ptr(), count.data_ptr(), T, E, 2, 1, tile_rows, len(table), _lib.current_stream()), "plan")
    _check_tiles(table[:int(count)].tolist(), torch.bincount(chosen.flatten(), minlength=E).tolist(), tile_rows)


def _check_tiles(table, counts, tile_rows):
    at, start = 0, 0
    for e, c in enumerate(counts):
        mine, end = table[at:at - (-c // tile_rows)], start + c
        at += len(mine)
        for group, first, rows, _ in mine:
            assert (group, first) == (e, start) and 0 < rows <= tile_rows
            start += rows
        assert start == end
    assert at == len(table)


@pytest.mark.parametrize("M, N", [(8, 8), (136, 264), (200, 520)])
def test_weight_gradient_has_the_same_bits_wherever_it_is_written(vb, M, N):
    """c on 16, 8 and 4 bytes: the tensor-core kernel serves all three."""
    from vexact_b200 import _lib

    lens = [5, 0, 64, 100]
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0)], dtype=torch.int32, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(M)
    a, b = (torch.randn(sum(lens), n, device="cuda", generator=gen).to(BF) for n in (M, N))
    size, got = len(lens) * M * N, []
    for at in (8, 12, 10):
        store = torch.full((size + 24,), 7.0, dtype=BF, device="cuda")
        _lib.check(_lib.load().b200_moe_grouped_wgrad(a.data_ptr(), b.data_ptr(), store.data_ptr() + 2 * at, cu.data_ptr(),
                                                      sum(lens), len(lens), M, N, _lib.current_stream()), "wgrad")
        assert (store[:at] == 7).all() and (store[at + size:] == 7).all()
        got.append(store[at:at + size])
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    refused = torch.empty(size + 8, dtype=BF, device="cuda")      # 2 bytes: neither kernel's accesses fit
    assert _lib.load().b200_moe_grouped_wgrad(a.data_ptr(), b.data_ptr(), refused.data_ptr() + 2, cu.data_ptr(), sum(lens),
                                              len(lens), M, N, _lib.current_stream()) == -2


@pytest.mark.parametrize("G, R, C", [(1, 8, 8), (3, 64, 72), (2, 200, 136)])
def test_transpose_of_the_last_two_dimensions(vb, G, R, C):
    """`b200_transpose_last2`, whole and partial 64 x 64 tiles."""
    from vexact_b200 import _lib

    x = torch.randint(-32768, 32767, (G, R, C), dtype=torch.int16, device="cuda")
    out = torch.empty(G, C, R, dtype=torch.int16, device="cuda")
    _lib.check(_lib.load().b200_transpose_last2(x.data_ptr(), out.data_ptr(), G, R, C, _lib.current_stream()), "transpose")
    assert torch.equal(out, x.transpose(1, 2))


@pytest.mark.parametrize("width", [8192, 8191])
def test_swiglu_rounds_every_bf16_gate_as_the_exact_form(width):
    """silu(g) of all 65536 bf16 values, in 16-byte and in 2-byte accesses, has torch's bits (NaN stays NaN), down to the
    values around -88 whose exponential is near the largest float and beyond, where it is infinite."""
    from vexact_b200 import _lib

    gate = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(BF).cuda()
    gate = torch.cat([gate, gate.new_zeros(-65536 % width)]).view(-1, width)
    one, out = torch.ones_like(gate), torch.empty_like(gate)
    _lib.check(_lib.load().b200_swiglu_scale(gate.data_ptr(), one.data_ptr(), None, out.data_ptr(), gate.shape[0], width,
                                             _lib.current_stream()), "swiglu")
    want = torch.nn.functional.silu(gate)
    assert torch.equal(out.isnan(), want.isnan())
    assert torch.equal(out.nan_to_num(0.0, float("inf"), -float("inf")).view(torch.int16),
                       want.nan_to_num(0.0, float("inf"), -float("inf")).view(torch.int16))


@pytest.mark.parametrize("M, N", [(8, 8), (128, 256), (136, 264), (200, 520), (768, 64)])
def test_grouped_weight_gradient_edges(M, N):
    """Groups of every length around the 16 rows of an instruction and the 64 of a step, empty ones between them; a group's
    NaN and infinities stay its own; rows of the operands may lie apart."""
    from vexact_b200 import _lib

    lens = [0, 1, 15, 16, 17, 0, 63, 64, 65, 200, 5, 0]
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0)], dtype=torch.int32, device="cuda")
    R, G = sum(lens), len(lens)
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    wide = torch.randn(R, 2 * M, device="cuda", generator=gen).to(BF)
    a, b = wide[:, M:], torch.randn(R, N, device="cuda", generator=gen).to(BF)
    bad = 10                                             # the group of five rows
    wide[cu[bad]:cu[bad + 1]] = float("nan")
    b[cu[bad]:cu[bad + 1]] = float("inf")

    def run():
        c = torch.full((G, M, N), 7.0, dtype=BF, device="cuda")
        _lib.check(_lib.load().b200_moe_grouped_wgrad_strided(a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), c.data_ptr(),
                                                              cu.data_ptr(), R, G, M, N, _lib.current_stream()), "wgrad")
        return c

    c = run()
    for g, n in enumerate(lens):
        if g == bad:
            assert torch.isnan(c[g]).all()
            continue
        s = slice(int(cu[g]), int(cu[g + 1]))
        ref = a[s].double().t() @ b[s].double()
        # one rounding to bf16 of an fp32 sum of n products of order 1
        torch.testing.assert_close(c[g].double(), ref, rtol=2 ** -8, atol=1e-6 * max(n, 1))
    assert torch.equal(c.nan_to_num(3.0), run().nan_to_num(3.0))


@pytest.mark.parametrize("K, N", [(64, 8), (72, 136), (192, 128), (768, 520)])
@pytest.mark.parametrize("tokens", [3, 130, 700])
def test_grouped_data_gradient_reads_weights_as_they_lie(K, N, tokens):
    """out = x @ w[g] with w [groups, K, N]: the bits of the forward form on the transposed weights, and both halves of a
    product in one accumulation when they come from two tensors."""
    from vexact_b200 import _lib, group_gemm as gg
    from vexact_b200.fused_moe import _permute

    E, k = 5, 2
    gen = torch.Generator(device="cuda").manual_seed(K + N + tokens)
    sel = torch.randint(0, E, (tokens, k), device="cuda", generator=gen)
    plan = _permute(sel, None, None, E)
    ends, R = plan["cu_seqlens"][1:], tokens * k
    x = torch.randn(R, K, device="cuda", generator=gen).to(BF)
    w = torch.randn(E, K, N, device="cuda", generator=gen).to(BF)
    out = gg.group_gemm_same_nk(x, w, ends, R, transpose_b=False)
    assert torch.equal(out, gg.group_gemm_same_nk(x, w.transpose(1, 2).contiguous(), ends, R, transpose_b=True))
    cu = plan["cu_seqlens"].tolist()
    ref = torch.cat([x[cu[e]:cu[e + 1]].double() @ w[e].double() for e in range(E)])
    tol = dict(rtol=2 ** -8, atol=1e-6 * K)
    torch.testing.assert_close(out.double(), ref, **tol)
    if K % 64:
        return
    x2 = torch.randn(R, 2 * K, device="cuda", generator=gen).to(BF)
    w2 = torch.randn(E, K, N, device="cuda", generator=gen).to(BF)

    def product(a, first, second):
        y = torch.empty(R, N, dtype=BF, device="cuda")
        _lib.check(_lib.load().b200_moe_grouped_dgrad(
            a.data_ptr(), first.data_ptr(), _lib.ptr(second), y.data_ptr(), plan["tile_table"].data_ptr(),
            plan["tile_count"].data_ptr(), R, E, N, a.shape[1], y.stride(0), plan["max_tiles"], plan["tile_rows"],
            _lib.current_stream()), "dgrad")
        return y

    assert torch.equal(product(x2, w, w2), product(x2, torch.cat([w, w2], 1), None))
    ref = torch.cat([x2[cu[e]:cu[e + 1]].double() @ torch.cat([w[e], w2[e]]).double() for e in range(E)])
    torch.testing.assert_close(product(x2, w, w2).double(), ref, **tol)


@pytest.mark.parametrize("T, N, K", [(1024, 64, 64), (1025, 67, 96), (517, 130, 2048), (70000, 1, 32)])
def test_fp32_products_in_groups_have_the_single_outputs_bits(vb, T, N, K):
    """Many outputs run 4 x 4 to eight lanes, few a warp each: the same partial sums joined in the same order."""
    from vexact_b200.batch_invariant_ops import linear_f32_from_bf16

    x, w = _seeded(T, K, seed=T).cuda(), _seeded(N, K, seed=N).cuda()
    many = linear_f32_from_bf16(x, w)
    for r in (slice(0, 1), slice(T // 2, T // 2 + 3), slice(T - 1, T)):
        assert torch.equal(many[r], linear_f32_from_bf16(x[r], w))
    # K fp32 products of order 1
    torch.testing.assert_close(many.double(), x.double() @ w.double().t(), rtol=1e-6, atol=2e-7 * K)
