"""Kernels at the edges of their tiles: one row more or less than a tile, the shortest inputs, views that only just qualify.

Tolerances: bf16 rounds to a relative error of at most u = 2^-9.  A result passes through at most four rounded tiles after its inputs
(an output) or eight (a gradient), each a sum of terms of the size of the result, so the relative Frobenius error is below 4u and 8u;
twice that leaves room for sums whose terms cancel."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from linear_moe_b200 import ops
from linear_moe_b200.ops import cuda as K
from linear_moe_b200.ref import lsm as RL
from linear_moe_b200.ref import ops as R

U = 2.0 ** -9
OUT, GRAD = 8 * U, 16 * U


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-12)).item()


def run(f, ins, gout):
    ins = [t.detach().clone().requires_grad_(True) for t in ins]
    out = f(*ins)
    out = out if isinstance(out, tuple) else (out,)
    torch.autograd.backward(out[: len(gout)], gout)
    return list(out), [t.grad for t in ins]


def rand(*shape, scale=0.5):
    return (scale * torch.randn(*shape, device="cuda")).bfloat16()


def check(got, want, names):
    for name, a, b, tol in zip(names, got[0] + got[1], want[0] + want[1], [OUT] * len(got[0]) + [GRAD] * len(got[1])):
        assert rel(a, b) < tol, (name, rel(a, b), tol)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Tq,Tk,window", [(1, 1, None), (127, 127, None), (128, 128, None), (129, 129, None), (255, 383, None), (257, 257, 128),
                                          (300, 300, 1), (513, 513, 129)])
def test_attention_tile_edges(D, Tq, Tk, window):
    from linear_moe_b200.ops import flash, gemm
    torch.manual_seed(0)
    q, kv, go = rand(2, Tq, 4, D, scale=1), rand(2, Tk, 2, 2 * D, scale=1), rand(2, Tq, 4, D, scale=1)
    k, v = kv.split(D, dim=-1)
    assert flash.supported(q, k, v, True, window)
    got = run(lambda q, k, v: flash.FlashAttention.apply(q, k, v, D ** -0.5, Tk - Tq, window), [q, k, v], [go])
    gemm.check_error()
    want = run(lambda q, k, v: R.softmax_attention(q, k, v, D ** -0.5, True, Tk - Tq, window), [t.float() for t in (q, k, v)], [go.float()])
    if max(Tk if window is None else window, 1) == 1:           # one key each: dq and dk are exactly zero
        for a, b in zip(got[1][:2], want[1][:2]):
            assert a.abs().max() < 16 * U and b.abs().max() < 1e-4
        got, want = (got[0], got[1][2:]), (want[0], want[1][2:])
    check(got, want, ["o"] + ["dq", "dk", "dv"][-len(got[1]):])


def test_attention_in_sections():
    """Sequences so long that only two of three heads share the L2: the kernels' order over tiles and heads goes section by section, the last of them
    with one head.  Gradients enter in three places, and with a window a slice around each of them is all that they depend on."""
    from linear_moe_b200.ops import flash, gemm
    torch.manual_seed(0)
    T, H, D, W, n = 50000, 3, 128, 200, 400
    q, k, v, go = rand(1, T, H, D, scale=1), rand(1, T, H, D, scale=1), rand(1, T, H, D, scale=1), torch.zeros(1, T, H, D, device="cuda").bfloat16()
    starts = (0, 24960, T - n)
    for lo in starts:
        go[:, lo:lo + n] = rand(1, n, H, D, scale=1)
    (o,), grads = run(lambda q, k, v: flash.FlashAttention.apply(q, k, v, D ** -0.5, 0, W), [q, k, v], [go])
    gemm.check_error()
    for lo in starts:
        a = max(0, lo - W)
        (want,), wg = run(lambda q, k, v: R.softmax_attention(q, k, v, D ** -0.5, True, 0, W), [t[:, a:lo + n].float() for t in (q, k, v)],
                          [go[:, a:lo + n].float()])
        check(([o[:, lo:lo + n]], [t[:, a:lo + n] for t in grads]), ([want[:, lo - a:]], wg), ["o", "dq", "dk", "dv"])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T", [1, 15, 63, 64, 65, 200])
def test_delta_rule_chunk_edges(D, T):
    torch.manual_seed(0)
    B, H = 2, 3
    q, k, v = rand(B, T, H, 3 * D).split(D, dim=-1)
    k = torch.nn.functional.normalize(k.float(), dim=-1).bfloat16()
    beta, g = torch.rand(B, T, H, device="cuda"), torch.nn.functional.logsigmoid(torch.randn(B, T, H, device="cuda") + 2)
    S0 = 0.2 * torch.randn(B, H, D, D, device="cuda")
    go, gS = rand(B, T, H, D, scale=1), 0.05 * torch.randn(B, H, D, D, device="cuda")
    ins = [q, k, v, beta, g, S0]
    got = run(lambda q, k, v, beta, g, S: ops.lsm_delta(q, k, v, beta, g, None, S, 64), ins, [go, gS])
    want = run(lambda q, k, v, beta, g, S: RL.recurrent_lsm(q, k, v, beta=beta, g=g, initial_state=S), [t.float() for t in ins], [go.float(), gS])
    check(got, want, ["o", "S", "dq", "dk", "dv", "dbeta", "dg", "dS0"])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T", [1, 64, 130, 320])
def test_delta_scans_of_padded_and_dense_tiles(D, T):
    """The tile kernel's padded rows (one bulk copy per tile) and dense tiles (copies by all threads) give the same bits."""
    torch.manual_seed(0)
    B, H = 1, 3
    q, v = rand(B, T, H, D), rand(B, T, H, D)
    k = torch.nn.functional.normalize(torch.randn(B, T, H, D, device="cuda"), dim=-1).bfloat16()
    tiles = K._delta_prepare_kernel(q, k, v, torch.rand(B, T, H, device="cuda"), None, D ** -0.5)
    assert tiles[0].stride(3) == D + 8
    dense = [t.contiguous() for t in tiles]
    go, outs = rand(B, T, H, D, scale=1), []
    for W, U_, Qd, Kd, A, gamma in (tiles, dense):
        o = torch.empty(B, T, H, D, dtype=torch.bfloat16, device="cuda")
        outs.append([o, *K._delta_scan_fwd(W, U_, Qd, Kd, A, gamma, None, o), *K._delta_scan_fwd(W, U_, Qd, Kd, A, gamma, None),
                     *K._delta_scan_bwd(W, Qd, Kd, A, gamma, go, None)])
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T", [2, 15, 17, 63, 64, 65, 129, 200])
def test_vector_decay_chunk_edges(D, T):
    torch.manual_seed(0)
    B, H = 2, 3
    q, k, v = rand(B, T, H, 3 * D).split(D, dim=-1)
    g = torch.nn.functional.logsigmoid(2 * torch.randn(B, T, H, D, device="cuda")) / 4
    S0, gS = 0.3 * torch.randn(B, H, D, D, device="cuda"), 0.1 * torch.randn(B, H, D, D, device="cuda")
    go = rand(B, T, H, D, scale=1)
    ins = [q, k, v, g, S0]
    got = run(lambda q, k, v, g, S: ops.lsm_vector(q, k, v, g, None, S, None, 64), ins, [go, gS])
    want = run(lambda q, k, v, g, S: RL.recurrent_lsm(q, k, v, gk=g, initial_state=S), [t.float() for t in ins], [go.float(), gS])
    check(got, want, ["o", "S", "dq", "dk", "dv", "dg", "dS0"])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,chunks", [(2, 2, 1), (2, 2, 2), (2, 2, 3), (2, 2, 4), (2, 2, 5), (2, 2, 7), (40, 4, 1), (40, 4, 3)])
def test_vector_decay_long_groups(B, H, chunks, D, monkeypatch):
    """A group that walks `chunks` chunks of 64 tokens and a shorter one behind it with a ragged tail: double-buffered tiles, sums and
    tables are used again.  160 sequences are more than an SM has CTAs of 64-wide heads.  The decays' gradient as in
    test_scalar_decay_above_the_line, per channel."""
    torch.manual_seed(0)
    T = 64 * (2 * chunks - 1) - 19 if chunks > 1 else 100
    G = -(-T // (64 * chunks))
    monkeypatch.setattr(K, "lsm_groups", lambda *a: (G, chunks))
    x, go = rand(B, T, H, 3 * D), rand(B, T, H, D, scale=1)
    g = torch.nn.functional.logsigmoid(2 * torch.randn(B, T, H, D, device="cuda")) / 4
    S0 = 0.3 * torch.randn(B, H, D, D, device="cuda")
    got = run(lambda x, g, S: ops.lsm_vector(*x.split(D, dim=-1), g, None, S, None, 64), [x, g, S0], [go])
    want = run(lambda x, g, S: RL.recurrent_lsm(*x.split(D, dim=-1), gk=g, initial_state=S), [x.float(), g, S0], [go.float()])
    (dx, dg, dS), (wx, wg, wS) = got[1], want[1]
    check((got[0], [dx, dS]), (want[0], [wx, wS]), ["o", "S", "dqkv", "dS0"])
    q, k, _ = x.float().split(D, dim=-1)
    dq, dk, _ = wx.split(D, dim=-1)
    walk = ((q * dq).square() + (k * dk).square()).flip(1).cumsum(1).sqrt()
    assert (dg - wg).norm() < GRAD * walk.norm()


@pytest.mark.parametrize("h,f", [(128, 8), (200, 120), (256, 136), (512, 264)])
@pytest.mark.parametrize("counts", [[512, 0, 256], [0, 0, 768], [256, 1024, 0]])
def test_expert_mlp_epilogues(h, f, counts):
    """The activation and its gradient as epilogues of the grouped products: widths that end inside a tile, experts without rows."""
    from linear_moe_b200.ops import gemm
    torch.manual_seed(0)
    E, rows = len(counts), sum(counts)
    offs = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    assert all(c % gemm.ROW_ALIGN == 0 for c in counts)
    x, w1, w2, go = rand(rows, h, scale=1), rand(E, h, 2 * f, scale=h ** -0.5), rand(E, f, h, scale=f ** -0.5), rand(rows, h, scale=1)

    def plain(x, w1, w2):
        ys = []
        for e, xe in enumerate(x.split(counts)):
            gate, up = (xe @ w1[e]).chunk(2, dim=-1)
            ys.append((torch.nn.functional.silu(gate) * up) @ w2[e])
        return torch.cat(ys)
    got = run(lambda x, w1, w2: gemm.expert_mlp(x, w1, w2, offs), [x, w1, w2], [go])
    gemm.check_error()
    want = run(plain, [t.float() for t in (x, w1, w2)], [go.float()])
    check(got, want, ["y", "dx", "dw1", "dw2"])


@pytest.mark.parametrize("sms", [2, 6])
@pytest.mark.parametrize("h,f", [(200, 120), (256, 264), (512, 136)])
@pytest.mark.parametrize("counts", [[512, 0, 256, 0, 1024, 256], [0, 768, 0, 0, 256, 512]])
def test_expert_mlp_many_tiles_per_pair(h, f, counts, sms, monkeypatch):
    """One or three CTA pairs for all tiles: the search for the next tile's expert goes on from the last one, gate and up values are requested
    for the next tile, both accumulator buffers are used again.  The same bits as with a pair per tile, and right."""
    from linear_moe_b200.ops import gemm
    torch.manual_seed(0)
    E, rows = len(counts), sum(counts)
    offs = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    assert rows // 256 * -(-f // 128) > sms // 2 and rows // 256 * -(-h // 256) > sms // 2      # tiles of the products
    x, w1, w2, go = rand(rows, h, scale=1), rand(E, h, 2 * f, scale=h ** -0.5), rand(E, f, h, scale=f ** -0.5), rand(rows, h, scale=1)

    def kernel():
        y, g = run(lambda x, w1, w2: gemm.expert_mlp(x, w1, w2, offs), [x, w1, w2], [go])
        gemm.check_error()
        return y, g
    whole = kernel()
    monkeypatch.setattr(K, "NUM_SMS", sms)
    got = kernel()
    for a, b in zip(got[0] + got[1], whole[0] + whole[1]):
        assert torch.equal(a, b)

    def plain(x, w1, w2):
        ys = []
        for e, xe in enumerate(x.split(counts)):
            gate, up = (xe @ w1[e]).chunk(2, dim=-1)
            ys.append((torch.nn.functional.silu(gate) * up) @ w2[e])
        return torch.cat(ys)
    check(got, run(plain, [t.float() for t in (x, w1, w2)], [go.float()]), ["y", "dx", "dw1", "dw2"])


@pytest.mark.parametrize("T", [2, 127, 128, 129, 400])
@pytest.mark.parametrize("decay", ["none", "head", "token"])
@pytest.mark.parametrize("layout", ["fused", "heads first", "shared keys"])
def test_scalar_decay_wide_chunks(T, decay, layout, monkeypatch):
    """128-wide heads in chunks of 128 tokens (decays that are not trained), over the strides that callers come with."""
    from linear_moe_b200.ops import gemm
    torch.manual_seed(0)
    B, H, D = 2, 3, 128
    g = {"none": None, "head": -torch.tensor([0.002, 0.1, 1.5], device="cuda"), "token": -0.3 * torch.rand(B, T, H, device="cuda")}[decay]
    q, k, v = rand(B, T, H, 3 * D).split(D, dim=-1)
    if layout == "heads first":
        q, k, v = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v))
    elif layout == "shared keys":
        k, v = k[:, :, :1].expand(-1, -1, H, -1), v[:, :1, :1].expand(-1, T, H, -1)
    S0, gS = 0.3 * torch.randn(B, H, D, D, device="cuda"), 0.1 * torch.randn(B, H, D, D, device="cuda")
    go = rand(B, T, H, D, scale=1)
    monkeypatch.setattr(K, "_scalar_chunk", lambda *a: 128)       # the rule takes longer inputs only

    def kernel(q, k, v, S):
        return ops.lsm_scalar(q, k, v, g, None, S, 64)

    def ref(q, k, v, S):
        gt = None if g is None else (g.expand(B, T, H) if g.dim() == 1 else g)
        return RL.recurrent_lsm(q, k, v, g=gt, initial_state=S)
    got, want = [], []
    for f, ins, res in ((kernel, (q, k, v, S0), got), (ref, [t.float() for t in (q, k, v, S0)], want)):
        ins = [t.detach().requires_grad_(True) for t in ins]
        out = f(*ins)
        res += [list(out), list(torch.autograd.grad(out, ins, [go.to(out[0].dtype), gS]))]
    gemm.check_error()
    check(got, want, ["o", "S", "dq", "dk", "dv", "dS0"])
    with torch.no_grad():
        o, S = kernel(q, k, v, S0)
    assert torch.equal(o, got[0][0]) and torch.equal(S, got[0][1])


@pytest.mark.parametrize("chunks", [1, 2, 3, 4, 5, 7])
@pytest.mark.parametrize("decay", ["head", "token"])
def test_scalar_decay_wide_chunks_in_long_groups(chunks, decay, monkeypatch):
    """A group that walks `chunks` chunks of 128 tokens and a shorter one behind it with a ragged tail: stages, barrier phases and output
    buffers are used again, the state and the running decays go from chunk to chunk and from group to group."""
    from linear_moe_b200.ops import gemm
    torch.manual_seed(0)
    B, H, D, T = 2, 2, 128, 128 * (2 * chunks - 1) - 37 if chunks > 1 else 200
    G = -(-T // (128 * chunks))
    g = -torch.tensor([0.002, 0.1], device="cuda") if decay == "head" else -0.1 * torch.rand(B, T, H, device="cuda")
    monkeypatch.setattr(K, "_scalar_chunk", lambda *a: 128)
    monkeypatch.setattr(K, "_scalar_groups", lambda *a: (G, 2 * chunks))
    x = rand(B, T, H, 3 * D)
    S0, gS = 0.3 * torch.randn(B, H, D, D, device="cuda"), 0.1 * torch.randn(B, H, D, D, device="cuda")
    go = rand(B, T, H, D, scale=1)
    got = run(lambda x, S: ops.lsm_scalar(*x.split(D, dim=-1), g, None, S, 64), [x, S0], [go, gS])
    gemm.check_error()
    want = run(lambda x, S: RL.recurrent_lsm(*x.split(D, dim=-1), g=g.expand(B, T, H), initial_state=S), [x.float(), S0], [go.float(), gS])
    check(got, want, ["o", "S", "dqkv", "dS0"])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("init", [True, False])
def test_trained_constant_decays(D, fused, init):
    """A log decay per head gets its gradient from one fused projection as well as from three tensors, with a trained initial state and
    without.  Its gradient is a sum over all tokens of differences of two gradients of GRAD each, here of the result's size."""
    torch.manual_seed(0)
    B, T, H = 2, 100, 3
    x, go = rand(B, T, H, 3 * D), rand(B, T, H, D, scale=1)
    g, S0 = -torch.tensor([0.02, 0.1, 0.4], device="cuda"), 0.3 * torch.randn(B, H, D, D, device="cuda")

    def kernel(x, g, *S):
        q, k, v = x.split(D, dim=-1)
        if not fused:
            q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
        return ops.lsm_scalar(q, k, v, g, None, *S)[0]

    def ref(x, g, *S):
        return RL.recurrent_lsm(*x.split(D, dim=-1), g=g.expand(B, T, H), initial_state=S[0] if S else None)[0]
    ins = [x, g] + [S0] * init
    got, want = run(kernel, ins, [go]), run(ref, [t.float() for t in ins], [go.float()])
    check(([], got[1]), ([], want[1]), ["dqkv", "dg", "dS0"][:len(ins)])


@pytest.mark.parametrize("decay", ["head", "token"])
@pytest.mark.parametrize("B,T,H", [(1, 9500, 16), (3, 200, 256), (1, 38001, 4)])
def test_scalar_decay_above_the_line(B, T, H, decay):
    """The wide chunks as the rule takes them, over several waves of groups, with trained decays: outputs and gradients against the chunked
    recurrence in 64 bits, and the same bits in training and in evaluation.  A log decay's gradient at t is the sum over i >= t of
    q_i . dq_i - k_i . dk_i, whose products carry independent relative errors of GRAD at most: a random walk of that step."""
    torch.manual_seed(0)
    D = 128
    assert K._scalar_chunk(B, T, H, D) == 128
    x, go = rand(B, T, H, 3 * D), rand(B, T, H, D, scale=1)
    a = torch.linspace(-4, 0, H, device="cuda")
    a = (a if decay == "head" else a + torch.randn(B, T, H, device="cuda")).requires_grad_(True)
    x1 = x.clone().requires_grad_(True)

    def f(x, a):
        q, k, v = x.split(D, dim=-1)
        return ops.lsm_scalar(q, k, v, -torch.exp(a), None, None, 64)
    o, S = f(x1, a)
    dx, da = torch.autograd.grad(o, [x1, a], go)
    with torch.no_grad():
        o2, S2 = f(x, a)
    assert torch.equal(o, o2) and torch.equal(S, S2)
    for h in range(0, H, max(1, H // 4)):                       # four heads: the recurrence in 64 bits is slow
        xs = x[:, :, h].double().requires_grad_(True)
        ah = (a[h] if decay == "head" else a[..., h]).detach().double().requires_grad_(True)
        g = -torch.exp(ah)
        q, k, v = xs.split(D, dim=-1)
        want, state = chunked64(q * D ** -0.5, k, v, g.expand(B, T))
        dxs, dah = torch.autograd.grad(want, [xs, ah], go[:, :, h].double())
        assert rel(o[:, :, h], want) < OUT and rel(S[:, h], state) < OUT and rel(dx[:, :, h], dxs) < GRAD
        dq, dk, _ = dxs.split(D, dim=-1)
        step = ((q * dq).square() + (k * dk).square()).sum(-1).detach()                               # [B, T]
        if decay == "token":
            walk = step.flip(1).cumsum(1).flip(1).sqrt()
        else:                                                   # the term of token i is in the sums of tokens 0 .. i
            walk = (step * torch.arange(1, T + 1, device="cuda").double().square()).sum().sqrt()
        assert (da[..., h] - dah).norm() < GRAD * (walk * g.detach()).norm()


def test_long_model_against_64_bits():
    """Loss and every weight's gradient of a two-layer model whose scans take the wide chunks by the rule.  The tolerance is the one of whole models
    in perf/cases.py; measured 0.016 (geometric mean over the weights) and 0.02 (largest)."""
    from perf import cases
    case = dict(kind="train", B=1, T=38016, layers=2, hidden=512, ffn=1024, vocab=1000)
    assert K._scalar_chunk(1, case["T"], case["hidden"] // 128, 128) == 128
    got, want = cases.run(cases.prepare(case, 1)), cases.exact(case, 1)
    for a, b in zip([got["loss"], *got["grads"]], [want["loss"], *want["grads"]]):
        assert rel(a, b) < cases.tolerance(case)["rel"]


def chunked64(q, k, v, g, C=100):
    """The scalar-decay recurrence for one head [B, T, D], decays [B, T], C tokens at a time."""
    S, out = q.new_zeros(q.shape[0], q.shape[-1], v.shape[-1]), []
    for t in range(0, q.shape[1], C):
        Q, K_, V, b = q[:, t:t + C], k[:, t:t + C], v[:, t:t + C], g[:, t:t + C].cumsum(1)
        decays = (b[:, :, None] - b[:, None, :]).tril().exp().tril()
        out.append(((Q @ K_.mT) * decays) @ V + b.exp()[..., None] * (Q @ S))
        S = b[:, -1].exp()[:, None, None] * S + (K_ * (b[:, -1:] - b).exp()[..., None]).mT @ V
    return torch.cat(out, 1), S


@pytest.mark.parametrize("kind,D", [("scalar", 64), ("scalar", 128), ("vector", 64), ("vector", 128), ("delta", 128)])
@pytest.mark.parametrize("T", [2, 200])
def test_forward_in_one_host_call(kind, D, T):
    """Without gradients the forward pass goes past the autograd function: same bits, and not inside a transform."""
    torch.manual_seed(0)
    B, H = 2, 3
    q, k, v = rand(B, T, H, 3 * D).split(D, dim=-1)
    g = -0.3 * torch.rand((B, T, H, D) if kind == "vector" else (B, T, H), device="cuda")
    S0 = 0.3 * torch.randn(B, H, D, D, device="cuda")
    f = {"scalar": lambda q: ops.lsm_scalar(q, k, v, g, None, S0, 64), "vector": lambda q: ops.lsm_vector(q, k, v, g, None, S0, None, 64),
         "delta": lambda q: ops.lsm_delta(q, k, v, -g, g, None, S0, 64)}[kind]
    want = f(q.detach().requires_grad_(True))
    with torch.no_grad():
        assert K._plain_call()
        got = f(q)
        with torch.autograd.forward_ad.dual_level():
            assert not K._plain_call()
        torch.func.vmap(lambda x: (x, assert_not_plain())[0])(torch.zeros(2))
        torch.jit.trace(lambda x: (x + 1, assert_not_plain())[0], torch.zeros(2), check_trace=False)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert not K._plain_call()


def assert_not_plain():
    assert not K._plain_call()


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,k", [(1, 32), (17, 2048), (130, 2080), (5000, 2048), (5000, 2304), (4752, 96), (300, 8192), (300, 8320), (20000, 288)])
def test_weight_streaming_edges(M, N, k):
    """Row blocks walked by two CTAs per SM or split over a cluster; x held in registers or not; K that ends inside a step."""
    torch.manual_seed(0)
    x, w = rand(M, k + 8, scale=1)[:, :k], rand(N, k, scale=k ** -0.5)
    assert K._skinny_ok(x, w)
    y = K.linear_skinny(x, w)
    assert rel(y, x.double() @ w.double().t()) < OUT
    acc = torch.randn(M, N, device="cuda")
    want = acc.double() + x.double() @ w.double().t()
    K._skinny_f32(x, w, acc, True)
    assert rel(acc, want) < 1e-5                                # fp32 sums of exact products: sqrt(K) 2^-24, K up to 8320


@pytest.mark.parametrize("M,k,few,many", [(8, 2048, 4736, 4752), (16, 4096, 4736, 4752), (3, 2560, 4736, 8192), (8, 4224, 1024, 5400), (16, 4224, 1024, 2064),
                                          (16, 8192, 512, 2048), (8, 9088, 1024, 2400), (8, 11008, 2368, 2384), (5, 96, 4000, 4800)])
def test_weight_streaming_routes(M, k, few, many):
    """A CTA per row block or row blocks walked with copies across their ends: the rule takes one for `few` rows of W and, for most of these, the
    other for `many`, and the columns that both have are the same bits where K is split alike (else within the rounding of a result)."""
    torch.manual_seed(0)
    x, w = rand(M, k, scale=1), rand(many, k, scale=k ** -0.5)
    a, b = K.linear_skinny(x, w[:few]), K.linear_skinny(x, w)
    split = [(n + 15) // 16 < 2 * K.num_sms() and k % 128 == 0 for n in (few, many)]
    assert torch.equal(a, b[:, :few]) if split[0] == split[1] else rel(a, b[:, :few]) < OUT
    assert rel(b, x.double() @ w.double().t()) < OUT
    for n in (few, many):
        assert torch.equal(K.linear_skinny_swiglu(x, w[:n]), K.swiglu(K.linear_skinny(x, w[:n])))


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("F,K_", [(8, 32), (24, 2048), (2504, 2048), (2400, 4096), (5000, 96)])
def test_weight_streaming_swiglu(M, F, K_):
    """The activation in the weight-streaming product gives the bits of the two launches it replaces."""
    torch.manual_seed(0)
    x, w = rand(M, K_, scale=1), rand(2 * F, K_, scale=2 * K_ ** -0.5)
    assert torch.equal(K.linear_skinny_swiglu(x, w), K.swiglu(K.linear_skinny(x, w)))


def test_early_launches_wait():
    """Chains of kernels that may start while the one before them runs: every link reads what the one before has written."""
    torch.manual_seed(0)
    n, h, H, D = 8, 1024, 8, 128
    w = [rand(h, h, scale=h ** -0.5) for _ in range(8)]
    gain, S0 = torch.ones(h, device="cuda").bfloat16(), torch.randn(n, H, D, D, device="cuda")
    wide = [torch.cat([m, m]) for m in w]
    x = rand(n, h, scale=1)

    def chain(pause):
        y, S = x, S0
        with torch.no_grad():
            for m, m2 in zip(w, wide):
                y = K.linear_skinny(y, m); pause()
                y = K.rms_norm(y, gain); pause()
                o, S = K.lsm_scalar(*(y.view(n, 1, H, D),) * 3, None, 0.05, S, 64); pause()
                y = K.head_norm_gate(o, gain[:D], y.view(n, 1, H, D), 1e-6, True).reshape(n, h); pause()
                y = K.linear_skinny_swiglu(y, m2); pause()
        return y, S
    want = chain(torch.cuda.synchronize)
    for _ in range(20):
        for a, b in zip(chain(lambda: None), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("V", [8, 4104, 32000, 65544])
def test_cross_entropy_rows(V):
    """Loss and softmax - onehot in one pass over the logits: fewer pieces than threads, ragged last rounds, ignored rows, a row of equal logits."""
    torch.manual_seed(0)
    x = rand(37, V, scale=3)
    x[5] = 1.5
    labels = torch.randint(0, V, (37,), device="cuda")
    labels[3], labels[9] = -100, V - 1
    z, loss = x.clone(), torch.empty(37, device="cuda")
    K.softmax_ce_rows(z, labels, loss, -100)
    ref = x.double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(ref, labels, ignore_index=-100, reduction="none")
    g, = torch.autograd.grad(want.sum(), ref)
    torch.testing.assert_close(loss.double(), want.detach(), rtol=1e-5, atol=1e-5)          # fp32 sums and exponentials
    torch.testing.assert_close(z.double(), g, rtol=2 ** -8, atol=1e-6)                     # one rounding to bf16


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,V,h", [(1, 8, 8), (300, 1000, 264), (500, 1000, 1032)])
def test_embedding_gradient_of_few_tokens(T, V, h, dtype):
    """The dense gradient of a table, with ids that are their token's own, shared by two and by many tokens, and outside this shard of the table."""
    torch.manual_seed(0)
    w = torch.randn(V, h, device="cuda", dtype=dtype).requires_grad_(True)
    ids = torch.randint(100, 100 + V, (T,), device="cuda")
    if T > 1:
        ids[: T // 3] = 100 + V - 1
        ids[-1], ids[-2] = 3, 100 + V + 7
    go = torch.randn(T, h, device="cuda", dtype=dtype)
    got, = torch.autograd.grad(K.embedding(ids, w, 100, True), w, go)
    inside = (ids >= 100) & (ids < 100 + V)
    want = torch.zeros(V, h, device="cuda", dtype=torch.float64).index_add_(0, ids[inside] - 100, go[inside].double())
    assert got.dtype == dtype and rel(got, want) < (U if dtype == torch.bfloat16 else 1e-6)


def test_scaled_rows():
    x, h, g = rand(13, 1032, scale=1), rand(13, 1032, scale=1), rand(13, scale=1)
    wx, wh = x * g[:, None], h * g[:, None]
    a, b = K.scale_rows(x, h, g)
    assert a is x and torch.equal(a, wx) and torch.equal(b, wh)


@pytest.mark.parametrize("kind", ["scalar", "vector", "delta"])
def test_states_that_may_be_overwritten(kind):
    """One-token steps: a new state beside the old one, or over a state that was given away for that, with the same bits."""
    from linear_moe_b200.infer.generation import _overwritable
    torch.manual_seed(0)
    B, H, D = 3, 2, 128
    q, k, v = rand(B, 1, H, D), torch.nn.functional.normalize(torch.randn(B, 1, H, D, device="cuda"), dim=-1).bfloat16(), rand(B, 1, H, D)
    g, gk, beta = -torch.rand(B, 1, H, device="cuda"), -torch.rand(B, 1, H, D, device="cuda"), torch.rand(B, 1, H, device="cuda")
    step = {"scalar": lambda S: ops.lsm_scalar(q, k, v, g, None, S), "vector": lambda S: ops.lsm_vector(q, k, v, gk, None, S),
            "delta": lambda S: ops.lsm_delta(q, k, v, beta, g, None, S)}[kind]
    with torch.no_grad():
        S = torch.randn(B, H, D, D, device="cuda")
        before = S.clone()
        o, S1 = step(S)
        assert torch.equal(S, before) and S1.data_ptr() != S.data_ptr()
        o2, S2 = step(_overwritable(S))
        assert S2.data_ptr() == S.data_ptr() and torch.equal(S, S1) and torch.equal(o, o2)


@pytest.mark.parametrize("D", [64, 128])
def test_bonus_step_over_its_state(D):
    """One token with a bonus (RWKV6), whose output needs the state in front of it: the same bits beside the old state and over it, and as the
    definition has it."""
    from linear_moe_b200.infer.generation import _overwritable
    torch.manual_seed(0)
    B, H = 3, 2
    q, k, v, u = rand(B, 1, H, D), rand(B, 1, H, D), rand(B, 1, H, D), torch.randn(H, D, device="cuda")
    gk, S = -torch.rand(B, 1, H, D, device="cuda"), torch.randn(B, H, D, D, device="cuda")
    with torch.no_grad():
        o, S1 = ops.lsm_vector(q, k, v, gk, None, S, u)
        q0, k0, v0 = (t[:, 0].double() for t in (q, k, v))
        kv = k0[..., None] * v0[..., None, :]
        want = D ** -0.5 * torch.einsum("bhk,bhkv->bhv", q0, S.double() + u.double()[..., None] * kv)
        # three roundings to bf16: of the two terms and of their sum
        assert rel(o[:, 0], want) < 4 * U and rel(S1, gk[:, 0].double().exp()[..., None] * S.double() + kv) < 1e-5
        o2, S2 = ops.lsm_vector(q, k, v, gk, None, _overwritable(S), u)
        assert torch.equal(o, o2) and torch.equal(S1, S2)


@pytest.mark.parametrize("B,H,T", [(1, 9, 700), (2, 5, 700), (1, 149, 70)])
def test_vector_decay_views(B, H, T):
    """128-wide heads from views that tensor maps or 16-byte loads could not take as they are (heads that repeat one another, a value that starts 2 bytes
    behind a boundary, states 4 bytes behind one), with few and many sequences for the combine kernel: the same bits as from dense copies."""
    from linear_moe_b200.ops import gemm
    torch.manual_seed(0)
    D = 128
    q = rand(B, T, 1, D).expand(B, T, H, D)
    k = rand(B, T, H, 3 * D)[..., D:2 * D]
    v = rand(B * T * H * D + 1)[1:].view(B, T, H, D)
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, H, D, device="cuda")) / 4
    S0, gS = (torch.randn(B * H * D * D + 1, device="cuda")[1:].view(B, H, D, D) for _ in range(2))
    go = rand(B * T * H * D + 1, scale=1)[1:].view(B, T, H, D)
    outs = []
    for copy in (lambda t: t, lambda t: t.clone(memory_format=torch.contiguous_format)):
        ins = [copy(t).detach().requires_grad_(True) for t in (q, k, v, g, S0)]
        out = ops.lsm_vector(*ins[:4], None, ins[4], None, 64)
        outs.append([*out, *torch.autograd.grad(list(out), ins, [copy(go), copy(gS)])])
    gemm.check_error()
    for a, b in zip(*outs):
        assert torch.equal(a, b)


def test_vector_decay_repeats():
    """Sixteen chunks in a row on most SMs, several times: the same bits.  (Two sets of warps take turns with the stages of a ring.)"""
    torch.manual_seed(0)
    B, T, H, D = 8, 2048, 8, 128
    x, go = rand(B, T, H, 3 * D), rand(B, T, H, D, scale=1)
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, H, D, device="cuda")) / 4
    first = None
    for _ in range(6):
        (o, S), grads = run(lambda x, g: ops.lsm_vector(*x.split(D, dim=-1), g, None, None, None, 64), [x, g], [go])
        first = first or [o, S, *grads]
        for a, b in zip(first, [o, S, *grads]):
            assert torch.equal(a, b)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,H", [(1, 1, 1), (2, 127, 3), (1, 129, 2), (1, 1024, 3), (1, 1025, 3), (3, 2500, 7), (1, 2049, 3)])
def test_decay_gradient_sums(B, T, H, D):
    """Sums from a token to the end, of a cluster in one round or several and of two launches, against 64 bits: n terms of up to three roundings
    each, added in any order, are off by (n + 3) units of their absolute sum at most."""
    torch.manual_seed(0)
    qkv, d = rand(B, T, H, 3 * D, scale=1), rand(B, T, H, 3 * D, scale=1)
    q, k, dq, dk = qkv[..., :D], qkv[..., D:2 * D], d[..., :D], d[..., D:2 * D]
    got = K._gla_dg(q, k, dq, dk).double()
    a, b = q.double() * dq.double(), k.double() * dk.double()
    want, size = ((x.flip(1).cumsum(1).flip(1)) for x in (a - b, a.abs() + b.abs()))
    assert ((got - want).abs() <= (T + 3) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("B,T,H,dv", [(2, 300, 2, 32), (2, 300, 2, 64), (1, 150, 60, 96), (1, 150, 75, 64), (1, 130, 25, 192), (2, 300, 32, 128), (1, 2050, 2, 128), (1, 64, 149, 128)])
def test_delta_rule_sizes(B, T, H, dv):
    """128-wide keys with other value widths (multiples of 64 on the 5th-generation tensor cores, with many heads or chunks), and more chunks than SMs: the
    kernel of the tiles' gradients goes on to a next chunk while it works on one."""
    from linear_moe_b200.ops import gemm
    torch.manual_seed(0)
    D = 128
    q, k = rand(B, T, H, D), torch.nn.functional.normalize(torch.randn(B, T, H, D, device="cuda"), dim=-1).bfloat16()
    v, beta = rand(B, T, H, dv), torch.rand(B, T, H, device="cuda")
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, H, device="cuda") + 2)
    S0, go, gS = 0.2 * torch.randn(B, H, D, dv, device="cuda"), rand(B, T, H, dv, scale=1), 0.05 * torch.randn(B, H, D, dv, device="cuda")
    ins = [q, k, v, beta, g, S0]
    got = run(lambda q, k, v, beta, g, S: ops.lsm_delta(q, k, v, beta, g, None, S, 64), ins, [go, gS])
    gemm.check_error()
    want = run(lambda q, k, v, beta, g, S: RL.recurrent_lsm(q, k, v, beta=beta, g=g, initial_state=S), [t.float() for t in ins], [go.float(), gS])
    check(got, want, ["o", "S", "dq", "dk", "dv", "dbeta", "dg", "dS0"])


def test_delta_prompt_repeats():
    """Forward calls without gradients, chains of 33 and 34 chunks on most SMs, several times: the same bits, and every wait came to its end.  (Outputs are
    stored by a warp of their own, from a ring of stages.)"""
    from linear_moe_b200.ops import gemm
    torch.manual_seed(0)
    B, H, D = 4, 18, 128
    for T in (2100, 2176):
        q, k = rand(B, T, H, D), torch.nn.functional.normalize(torch.randn(B, T, H, D, device="cuda"), dim=-1).bfloat16()
        v, beta = rand(B, T, H, D), torch.rand(B, T, H, device="cuda")
        with torch.no_grad():
            o, S = ops.lsm_delta(q, k, v, beta, None, None, None, 64)
            for _ in range(8):
                o2, S2 = ops.lsm_delta(q, k, v, beta, None, None, None, 64)
                assert torch.equal(o, o2) and torch.equal(S, S2)
        gemm.check_error()


@pytest.mark.parametrize("H,N,dv,tc", [(2, 31, 128, ""), (2, 32, 128, "output reverse"), (37, 40, 128, "output reverse"), (38, 3, 128, "output states reverse"),
                                       (50, 2, 96, ""), (50, 2, 192, "output states reverse")])
def test_delta_scan_routes(H, N, dv, tc):
    """Which scans of 128-wide keys run on tcgen05: those with outputs and the reverse one from 32 chunks on, those that only rebuild the increments and
    states (a step with few heads takes longer there) where the CTAs of the others are more than SMs.  Both give the increments and states of the definition."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines go by 148 SMs")
    torch.manual_seed(0)
    D = 128
    kw = dict(device="cuda", dtype=torch.bfloat16)
    W, Qd, Kd = (0.05 * torch.randn(1, H, N, 64, D, **kw) for _ in range(3))              # small enough for roundings to fade over the chunks
    U, A, dO = torch.randn(1, H, N, 64, dv, **kw), 0.1 * torch.randn(1, H, N, 64, 64, **kw).tril(), torch.randn(1, N * 64, H, dv, **kw)
    gamma, o = torch.full((1, H, N), 0.5, device="cuda"), torch.empty(1, N * 64, H, dv, **kw)
    calls = {"output": lambda: K._delta_scan_fwd(W, U, Qd, Kd, A, gamma, None, o, keep=False), "states": lambda: K._delta_scan_fwd(W, U, Qd, Kd, A, gamma, None),
             "reverse": lambda: K._delta_scan_bwd(W, Qd, Kd, A, gamma, dO, None)}
    for name, f in calls.items():
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
            res = f()
            torch.cuda.synchronize()
        scans = [e.key for e in p.key_averages() if "delta_scan" in e.key]
        assert len(scans) == 1 and ("_tc_kernel" in scans[0]) == (name in tc.split()), (name, scans)
        if name == "states":
            S = torch.zeros(1, H, D, dv, dtype=torch.float64, device="cuda")
            for n in range(N):
                vn = U[:, :, n].double() - W[:, :, n].double() @ S
                assert n == 0 or rel(res[1][:, :, n], S) < 8 * 2.0 ** -9
                assert rel(res[0][:, :, n], vn) < 8 * 2.0 ** -9
                S = 0.5 * S + Kd[:, :, n].double().transpose(-1, -2) @ vn


@pytest.mark.parametrize("B,H,T,chunks", [(1, 9, 700, 4), (2, 5, 700, 11), (1, 149, 130, 3)])
def test_vector_decay_views_in_groups(B, H, T, chunks, monkeypatch):
    """As test_vector_decay_views, in groups of several chunks (the tcgen05 kernels)."""
    monkeypatch.setattr(K, "lsm_groups", lambda *a: (-(-T // (64 * chunks)), chunks))
    test_vector_decay_views(B, H, T)


@pytest.mark.parametrize("B,T,H,D,tc", [(1, 2, 1, 128, False), (1, 64 * 74, 2, 128, False), (1, 64 * 74 + 1, 2, 128, True), (150, 64, 1, 128, False),
                                        (150, 65, 1, 128, True), (2, 64 * 200, 1, 64, False)])
def test_vector_decay_routes(B, T, H, D, tc):
    """128-wide heads run on tcgen05 where a group has several chunks, forward and backward; a call with one chunk per group does not pay for tensor maps and
    the later start."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the line goes by 148 SMs")
    torch.manual_seed(0)
    ins = [rand(B, T, H, D).requires_grad_(True) for _ in range(3)] + [-torch.rand(B, T, H, D, device="cuda").requires_grad_(True)]
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        o, _ = ops.lsm_vector(*ins, None, None, None, 64)
        torch.autograd.grad(o, ins, torch.ones_like(o))
        torch.cuda.synchronize()
    names = [e.key for e in p.key_averages() if "gla_" in e.key and "combine" not in e.key and "gla_dg" not in e.key]
    assert len(names) == 5 and all(("_tc_kernel" in n) == tc for n in names), names
