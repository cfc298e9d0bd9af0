"""GPU parity: tcgen05 weight-streaming GEMM vs the CPU oracle and the reference's golden
fixtures, and bitwise row invariance across batch sizes
(reference: tests/batch_invariant_ops/test_matmul.py:27-46, test_batch_invariance.py:30-128)."""
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


def _close_bf16(got, want, k):
    # stated tolerance: one bf16 ulp (rtol 2^-7) plus fp32 accumulation-order noise for results
    # that cancel towards zero; and the vast majority of elements bit-identical
    torch.testing.assert_close(got.float(), want.float(), rtol=2 ** -7, atol=1e-6 * k ** 0.5 + 1e-5)
    assert (got == want).float().mean() > 0.98


def test_gemm_golden(vb):
    for c in load_golden("matmul"):
        a, w, bias = c["a"].cuda(), c["w"].cuda(), c["bias"].cuda()
        _close_bf16(vb.matmul_persistent(a, w.t()).cpu(), c["out"], a.shape[1])
        _close_bf16(vb.matmul_persistent(a, w.t(), bias).cpu(), c["out_bias"], a.shape[1])


@pytest.mark.parametrize("M,K,N", [(1, 2048, 6144), (7, 2048, 6144), (64, 2048, 6144), (256, 2048, 6144),
                                   (300, 768, 2048), (512, 4096, 2048), (5, 72, 40), (129, 1536, 576)])
def test_gemm_oracle(vb, M, K, N):
    x = _seeded(M, K, seed=1)
    w = _seeded(N, K, seed=2, std=0.02)
    ref = ops.matmul(x, w.t())
    out = vb.matmul_persistent(x.cuda(), w.cuda().t())
    _close_bf16(out.cpu(), ref, K)
    # row-major B ([K, N] contiguous) and fp32 output
    out2 = vb.matmul_persistent(x.cuda(), w.t().contiguous().cuda())
    assert torch.equal(out, out2)
    out32 = vb.linear(x.cuda(), w.cuda(), out_dtype=torch.float32)
    assert torch.equal(out32.to(BF), out)


def test_gemm_bias_fp32_before_cast(vb):
    x = _seeded(33, 1536, seed=3)
    w = _seeded(256, 1536, seed=4, std=0.02)
    b = _seeded(256, seed=5, std=0.5)
    ref = ops.matmul(x, w.t(), b)
    out = torch.addmm(b.cuda(), x.cuda(), w.cuda().t()) if False else vb.matmul_persistent(x.cuda(), w.cuda().t(), b.cuda())
    _close_bf16(out.cpu(), ref, 1536)


def test_gemm_row_invariance_sweep(vb):
    """Row i of X @ W^T is bit-identical for every batch size 1..512."""
    K, N = 2048, 6144
    x = _seeded(512, K, seed=6).cuda()
    w = _seeded(N, K, seed=7, std=0.02).cuda()
    full = vb.matmul_persistent(x, w.t())
    sizes = sorted(set([1, 2, 3, 7, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 300, 384,
                        511, 512] + list(range(1, 513, 37))))
    for m in sizes:
        part = vb.matmul_persistent(x[:m], w.t())
        assert torch.equal(part, full[:m]), f"rows differ between batch {m} and batch 512"
    # a row's result does not depend on its position in the batch either
    perm = torch.randperm(512, generator=torch.Generator().manual_seed(0)).cuda()
    assert torch.equal(vb.matmul_persistent(x[perm].contiguous(), w.t()), full[perm])


def test_gemm_large_m_prefill_shape(vb):
    x = _seeded(2048, 2048, seed=8)
    w = _seeded(1024, 2048, seed=9, std=0.02)
    out = vb.matmul_persistent(x.cuda(), w.cuda().t())
    ref = ops.matmul(x, w.t())
    _close_bf16(out.cpu(), ref, 2048)
    assert torch.equal(vb.matmul_persistent(x[:5].cuda(), w.cuda().t()), out[:5])


def test_aten_override_routes_linear(vb):
    lin = torch.nn.Linear(512, 384, bias=True).to(BF).cuda()
    x = _seeded(9, 512, seed=10).cuda()
    with vb.set_batch_invariant_mode(True):
        y = lin(x)
        y1 = lin(x[:1])
        lsm = torch.log_softmax(x.float(), dim=-1)
    assert torch.equal(y[:1], y1)
    _close_bf16(y.cpu(), ops.matmul(x.cpu(), lin.weight.detach().cpu().t(), lin.bias.detach().cpu()), 512)
    torch.testing.assert_close(lsm.cpu(), ops.log_softmax(x.float().cpu()), rtol=0, atol=6e-6)
    assert not vb.is_batch_invariant_mode_enabled()


def test_gemm_f32_router(vb):
    x = _seeded(40, 2048, seed=11, dtype=torch.float32)
    w = _seeded(64, 2048, seed=12, std=0.02, dtype=torch.float32)
    out = vb.matmul_persistent(x.cuda(), w.cuda().t())
    torch.testing.assert_close(out.cpu(), x @ w.t(), rtol=1e-5, atol=1e-5)
    assert torch.equal(vb.matmul_persistent(x[:3].cuda(), w.cuda().t()), out[:3])


def test_status_word_clean(vb):
    torch.cuda.synchronize()
    assert vb._lib.read_status()[0] == 0


@pytest.mark.gpu
def test_fused_lm_head_greedy_matches_two_kernel_path_and_is_batch_invariant():
    """lm_head -> greedy token + logprob without the logits tensor: same tokens as GEMM + greedy_logprob,
    log-probabilities within 2e-5, and a token's (token, logprob) are the same bits at batch 1 and 512."""
    import vexact_b200 as vb
    from vexact_b200.standalone_logprobs import greedy_token_and_logprob, lm_head_greedy

    g = torch.Generator().manual_seed(21)
    for (T, K, V) in [(512, 2048, 151936), (300, 512, 4097), (7, 256, 130)]:
        x = torch.randn(T, K, generator=g).to(BF).cuda()
        w = (torch.randn(V, K, generator=g) * 0.02).to(BF).cuda()
        tok, lp = lm_head_greedy(x, w)
        tok_ref, lp_ref = greedy_token_and_logprob(vb.linear(x, w))
        assert torch.equal(tok, tok_ref), f"{(T, K, V)}: {(tok != tok_ref).sum().item()} tokens differ"
        torch.testing.assert_close(lp, lp_ref, rtol=0, atol=2e-5)
        for sub in ([0], [T - 1], list(range(0, T, max(1, T // 5)))):
            t1, l1 = lm_head_greedy(x[sub].contiguous(), w)
            assert torch.equal(t1, tok[sub]) and torch.equal(l1, lp[sub]), f"{(T, K, V)}: rows {sub} depend on the batch"
    # a tie: two identical weight rows give identical logits; the lower vocabulary index wins
    w[100] = w[3]
    x1 = (w[3].float() * 50).to(BF)[None].contiguous()
    t1, _ = lm_head_greedy(x1, w)
    tr, _ = greedy_token_and_logprob(vb.linear(x1, w))
    assert t1.item() == tr.item()
    from vexact_b200 import _lib
    assert _lib.read_status()[0] == 0


def test_fp16_matmul_and_batch_invariance(vb):
    """matmul_persistent on fp16 tensors (the reference serves bf16, fp16 and fp32): fp32 accumulation, bias in
    fp32, one rounding to fp16; a row's bits do not depend on the batch it is computed in."""
    g = torch.Generator().manual_seed(12)
    for (M, K, N) in [(1, 2048, 768), (7, 512, 200), (64, 2048, 6144), (300, 1536, 256)]:
        a = (torch.randn(M, K, generator=g)).half()
        w = (torch.randn(N, K, generator=g) * 0.05).half()
        bias = torch.randn(N, generator=g).half()
        ad, wd, bd = a.cuda(), w.cuda(), bias.cuda()
        out = vb.matmul_persistent(ad, wd.t())
        outb = vb.matmul_persistent(ad, wd.t(), bd)
        assert out.dtype == torch.float16
        ref = a.double() @ w.double().t()
        for got, want in ((out, ref), (outb, ref + bias.double())):
            err = (got.cpu().double() - want).abs()
            tol = 2.0 ** -10 * want.abs().clamp(min=0.5)           # one fp16 ulp, with a floor for cancellation
            assert bool((err <= tol).all()), (M, K, N, float(err.max()))
        assert torch.equal(vb.matmul_persistent(ad[:1], wd.t(), bd), outb[:1])
        if M > 8:
            assert torch.equal(vb.matmul_persistent(ad[5:8], wd.t(), bd), outb[5:8])


def test_mm_under_the_mode_takes_any_layout(vb):
    """Under the mode switch every aten::mm / addmm on CUDA tensors lands here, not only nn.Linear: a reduction
    length that is no multiple of 8, a row-major right operand, operands sliced at an odd element offset.  The
    reference's Triton kernel takes any strides (batch_invariant_ops.py:54-156); here such operands go through
    zero-padded copies, which leaves every fp32 accumulation as it was: the padded-K result equals the result
    for the same numbers laid out at K + pad with explicit zeros, and rows stay batch-invariant."""
    a = _seeded(33, 77, seed=21).cuda()
    b = _seeded(77, 50, seed=22).cuda()                     # row-major [K, N], K = 77
    with vb.set_batch_invariant_mode(True):
        c = torch.mm(a, b)
        c1 = torch.mm(a[:1], b)
        cb = torch.addmm(_seeded(50, seed=23).cuda(), a, b)
    assert torch.equal(c[:1], c1)
    a_pad = torch.nn.functional.pad(a, (0, 3))
    b_pad = torch.nn.functional.pad(b, (0, 0, 0, 3))
    assert torch.equal(c, vb.matmul_persistent(a_pad, b_pad))
    _close_bf16(c.cpu(), ops.matmul(a.cpu(), b.cpu()), 77)
    _close_bf16(cb.cpu(), ops.matmul(a.cpu(), b.cpu(), _seeded(50, seed=23)), 77)
    big = _seeded(9 * 64 + 1, seed=24).cuda()
    odd = big[1:].view(9, 64)                               # K fine, data pointer off by one element
    w = _seeded(64, 32, seed=25).cuda()
    assert torch.equal(vb.matmul_persistent(odd, w), vb.matmul_persistent(odd.clone(), w))


def test_conv3d_under_the_mode_is_deterministic_and_batch_invariant(vb):
    """Reference tests/batch_invariant_ops/test_torch_conv3d.py:50-115 (the Qwen3-VL patch embedding, cuDNN off):
    ten identical runs, and sample 0 alone equal to sample 0 of the batch."""
    import torch.nn.functional as F

    cout, cin, kt, kh, kw, batch = 1024, 3, 2, 16, 16, 8
    d, h, w = kt * 2, kh * 2, kw * 2
    a = torch.linspace(-1.0, 1.0, batch * cin * d * h * w, dtype=BF, device="cuda").reshape(batch, cin, d, h, w)
    weight = torch.linspace(-1.0, 1.0, cout * cin * kt * kh * kw, dtype=BF, device="cuda").reshape(cout, cin, kt, kh, kw)
    bias = torch.linspace(-1.0, 1.0, cout, dtype=BF, device="cuda")
    cudnn_was = torch.backends.cudnn.enabled
    torch.backends.cudnn.enabled = False
    try:
        with vb.set_batch_invariant_mode(True):
            out1 = F.conv3d(a, weight, bias=bias, stride=(kt, kh, kw))
            for _ in range(10):
                assert torch.equal(out1, F.conv3d(a, weight, bias=bias, stride=(kt, kh, kw)))
            single = F.conv3d(a[:1], weight, bias=bias, stride=(kt, kh, kw))
        assert torch.equal(single, out1[:1])
    finally:
        torch.backends.cudnn.enabled = cudnn_was
        torch.use_deterministic_algorithms(False)


@pytest.mark.parametrize("T, N, K", [(3001, 2056, 2048), (2049, 4104, 1096), (1250, 6152, 1536), (1033, 136, 20000),
                                     (1000, 128, 64), (1001, 200, 64), (1023, 384, 320), (1300, 1000, 72), (2048, 2056, 128),
                                     (4097, 136, 2048), (1000, 2048, 200)])
def test_products_on_cta_pairs_have_the_single_ctas_bits(vb, T, N, K):
    """From 1000 tokens on a product may run on CTA pairs, where that saves enough, as in the first four sizes (the fourth
    gated alone) (odd and partial weight tiles, partial token tiles, K with and
    without whole 64-wide atoms): every token's bits are those of the same token in a narrow batch, plain, with bias and gated."""
    from vexact_b200 import _lib

    gen = torch.Generator(device="cuda").manual_seed(T + N + K)
    x, w = (torch.randn(r, K, device="cuda", generator=gen).to(torch.bfloat16) for r in (T, 2 * N))
    bias = torch.randn(N, device="cuda", generator=gen).to(torch.bfloat16)

    def gated(a):
        out = torch.empty(a.shape[0], N, dtype=torch.bfloat16, device="cuda")
        _lib.check(_lib.load().b200_gemm_swiglu(a.data_ptr(), w.data_ptr(), out.data_ptr(), a.shape[0], N, K, K, K, N,
                                                _lib.current_stream()), "b200_gemm_swiglu")
        return out

    for f in (lambda a: vb.linear(a, w[:N]), lambda a: vb.linear(a, w[:N], bias), gated):
        wide = f(x)
        for r in (slice(0, 3), slice(T // 2 - 40, T // 2 + 41), slice(T - 130, T)):
            assert torch.equal(wide[r], f(x[r]))
    ref = x.double() @ w[:N].double().t()
    torch.testing.assert_close(vb.linear(x, w[:N]).double(), ref, rtol=2 ** -8, atol=1e-6 * K)
    g, u = (x.double() @ w.double().t()).to(torch.bfloat16).double().chunk(2, 1)
    # three bf16 roundings after the products
    torch.testing.assert_close(gated(x).double(), torch.nn.functional.silu(g) * u, rtol=2 ** -6, atol=2 ** -6 * K ** 0.5)


@pytest.mark.parametrize("T, N, K", [(64, 128, 512), (16, 256, 2048), (1500, 512, 256)])
def test_second_operand_may_be_the_output_of_the_launch_before(vb, T, N, K):
    """`k = x @ w^T; s = q @ k^T`, and a norm's output as the second operand: nothing is read from k before the launch that
    makes it is over, however early the next launch starts.  k's storage holds the result for other inputs before each call."""
    gen = torch.Generator(device="cuda").manual_seed(T + N)
    w, gamma = torch.randn(K, K, device="cuda", generator=gen).to(BF), torch.ones(K, device="cuda", dtype=BF)
    q = torch.randn(T, K, device="cuda", generator=gen).to(BF)
    xs = [torch.randn(N, K, device="cuda", generator=gen).to(BF) for _ in range(8)]

    def chain(x):
        k = vb.linear(x, w)
        s = vb.linear(q, k)
        n = vb.batch_invariant_rms_norm(k, gamma, 1e-6)
        return s, vb.linear(q, n)

    def apart(x):
        out = []
        k = vb.linear(x, w)
        torch.cuda.synchronize()
        out.append(vb.linear(q, k))
        n = vb.batch_invariant_rms_norm(k, gamma, 1e-6)
        torch.cuda.synchronize()
        return out + [vb.linear(q, n)]

    want = [apart(x) for x in xs]
    torch.cuda.synchronize()
    got = [chain(x) for x in xs]
    for a, b in zip(got, want):
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    static = xs[0].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain(static)
    for x, b in zip(xs, want):
        static.copy_(x)
        graph.replay()
        assert torch.equal(out[0], b[0]) and torch.equal(out[1], b[1])


def test_copies_of_weights_are_not_read_early(vb, monkeypatch):
    """Inside a pass with settled weights, a weight that `linear` has to copy (rows or a base that 16-byte accesses do not fit, columns
    first) is the output of the launch before its product, which therefore runs as outside the pass."""
    from vexact_b200 import _lib

    lib, calls = _lib.load(), []

    class Recorder:
        def __getattr__(self, name):
            f = getattr(lib, name)
            if not name.startswith("b200_"):
                return f
            return lambda *a: (calls.append((name, a[0]) if name == "b200_settled_weights" else name), f(*a))[1]

    monkeypatch.setattr(_lib, "load", lambda recorder=Recorder(): recorder)
    x = torch.randn(3, 72, device="cuda").to(BF)
    w = torch.randn(40, 80, device="cuda").to(BF)
    on, off = (("b200_settled_weights", v) for v in (1, 0))
    for weight in (w[:, 4:76], w.view(-1)[1:1 + 40 * 72].view(40, 72), w[:, :72].t().contiguous().t()):
        a = x[:, :weight.shape[1]]
        calls.clear()
        with _lib.settled_weights():
            out = vb.linear(a, weight)
        assert calls == [on, off, "b200_gemm_bf16", on, off], calls
        torch.testing.assert_close(out.float(), a.float() @ weight.float().t(), rtol=2 ** -7, atol=2e-2)
        calls.clear()
        vb.linear(a, weight)
        assert calls == ["b200_gemm_bf16"]
    calls.clear()
    with _lib.settled_weights():
        vb.linear(x, w[:, :72])
    assert calls == [on, "b200_gemm_bf16", off]
