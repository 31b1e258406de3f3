"""The peer-memory MoE exchange kernels on one GPU (a one-rank workspace) against the permute / grouped-MLP / un-permute
definition in fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from linear_moe_b200.ref import ops as R


@pytest.mark.parametrize("T,k,E,hid,f,drop", [(1000, 2, 4, 256, 128, False), (333, 8, 16, 512, 64, True), (64, 1, 2, 128, 256, False)])
def test_fused_moe_one_rank(T, k, E, hid, f, drop):
    from linear_moe_b200.models.moe import permute, unpermute
    from linear_moe_b200.ops import gemm
    from linear_moe_b200.ops.moe_fused import fused_moe
    from linear_moe_b200.parallel import fused_comm
    dev = torch.device("cuda", 0)
    torch.manual_seed(3)
    ws = fused_comm.MoeWorkspace(None, E, hid, T * k + 256 * E, dev)
    h = torch.randn(T, hid, device=dev).to(torch.bfloat16)
    logits = torch.randn(T, E, device=dev)
    probs, idx = torch.topk(torch.softmax(logits, -1), k, dim=-1)
    if drop:
        dropped = torch.rand(T, k, device=dev) < 0.2
        idx = torch.where(dropped, torch.full_like(idx, -1), idx)
        probs = probs * (~dropped)
    w1 = (0.05 * torch.randn(E, hid, 2 * f, device=dev)).to(torch.bfloat16)
    w2 = (0.05 * torch.randn(E, f, hid, device=dev)).to(torch.bfloat16)
    go = torch.randn(T, hid, device=dev).to(torch.bfloat16)

    def run(fused):
        hh, pp = h.clone().requires_grad_(True), probs.clone().requires_grad_(True)
        a, b = w1.clone().requires_grad_(True), w2.clone().requires_grad_(True)
        if fused:
            out = fused_moe(hh, pp, idx, a, b, ws)
            out.backward(go)
        else:
            hf, af, bf = hh.float(), a.float(), b.float()
            permuted, order, counts = permute(hf, idx, E)
            y = R.grouped_mlp(permuted, counts, af, bf)
            out = unpermute(y, order, pp, T, k)
            out.backward(go.float())
        return out, hh.grad, pp.grad, a.grad, b.grad

    for rep in range(2):                                    # twice: epochs and buffer reuse
        got = run(True)
        torch.cuda.synchronize()
        fused_comm.check_status("moe test")
        gemm.check_error()
    ref = run(False)
    for name, x, y in zip(["out", "dh", "dprobs", "dw1", "dw2"], got, ref):
        x, y = x.float(), y.float()
        err, scale = (x - y).abs().max().item(), y.abs().max().item()
        assert err <= 3e-2 * scale + 1e-3, f"{name}: err {err:.3e} scale {scale:.3e}"


def test_bounded_wait_expiry_and_overflow_are_reported():
    """Failure reporting of the exchange kernels without faulting anything: (a) a pull that waits for an epoch nobody
    signals gives up after its spin limit, sets the status word and returns; (b) routing more rows to a rank than its
    receive buffer holds sets the status word and sends nothing.  The context stays usable afterwards."""
    import ctypes
    from linear_moe_b200.ops import cuda as K
    from linear_moe_b200.parallel import fused_comm
    from linear_moe_b200.train.watchdog import CommTimeout
    dev = torch.device("cuda", 0)
    E, hid, T, k = 4, 128, 64, 2
    ws = fused_comm.MoeWorkspace(None, E, hid, T * k + 256 * E, dev, spin_limit=2000)
    idx = torch.randint(0, E, (T, k), device=dev)
    route = ws.route(idx)
    torch.cuda.synchronize()
    fused_comm.check_status("clean")                                   # nothing wrong so far
    # (a) wait for an epoch that is never signalled: ~2000 polls of 64 ns, then status + return
    a = ws._args()
    a.epoch = ws.ep_pull + 5
    out = torch.empty(T, hid, dtype=torch.bfloat16, device=dev)
    w = torch.ones(T, k, dtype=torch.float32, device=dev)
    a.w, a.out, a.rows = w.data_ptr(), out.data_ptr(), 0
    a.dest_rank, a.dest_row = route.dest_rank.data_ptr(), route.dest_row.data_ptr()
    a.n_assign, a.k = T * k, k
    ws._run(5, a, "moe_pull")
    torch.cuda.synchronize()
    with pytest.raises(CommTimeout):
        fused_comm.check_status("expired wait")
    fused_comm.check_status("cleared")                                 # the status word was reset
    # (b) receive buffer too small for the routed rows
    small = fused_comm.MoeWorkspace(None, E, hid, 256, dev)
    r2 = small.route(torch.zeros(1024, k, dtype=torch.int64, device=dev))      # 2048 rows to expert 0, capacity 256
    torch.cuda.synchronize()
    assert int((r2.dest_rank >= 0).sum()) == 0                         # nothing is sent
    with pytest.raises(CommTimeout):
        fused_comm.check_status("overflow")
    # the context is intact: a normal exchange still works
    x = torch.randn(T, hid, device=dev).to(torch.bfloat16)
    recv = ws.push(x, route, None)
    torch.cuda.synchronize()
    fused_comm.check_status("after")
    assert torch.isfinite(recv[: int(route.offs[-1])].float()).all()


@pytest.mark.parametrize("T,k,E,hid", [(1, 1, 3, 8), (1023, 1, 64, 72), (512, 2, 5, 264), (700, 16, 40, 520), (1100, 12, 7, 64)])
def test_one_rank_exchange_kernels(T, k, E, hid):
    """Routing, push, combine and its gradients on one rank: around the 1024 assignments of a routing block, one expert with most of the rows and
    one with none, dropped pairs, more slots than the push takes at a time, rows of one and of odd numbers of 16-byte pieces."""
    from linear_moe_b200.ops import gemm
    from linear_moe_b200.parallel import fused_comm
    dev = torch.device("cuda", 0)
    torch.manual_seed(1)
    pad = gemm.ROW_ALIGN
    ws = fused_comm.MoeWorkspace(None, E, hid, T * k + pad * E, dev)
    idx = torch.where(torch.rand(T, k, device=dev) < 0.5, torch.randint(0, E - 1, (T, k), device=dev), torch.zeros((), dtype=torch.int64, device=dev))
    idx = torch.where(torch.rand(T, k, device=dev) < 0.1, torch.full_like(idx, -1), idx)                 # (expert E - 1 gets nothing)
    route = ws.route(idx)
    flat = idx.reshape(-1)
    count = torch.bincount(flat[flat >= 0], minlength=E)
    segs = torch.cat([count.new_zeros(1), ((count + pad - 1) // pad * pad).cumsum(0)])
    assert torch.equal(route.real.long(), count) and torch.equal(route.offs.long(), segs)
    rank_in = torch.empty_like(flat)                                                                      # a stable counting sort
    for e in range(E):
        m = flat == e
        rank_in[m] = torch.arange(int(m.sum()), device=dev)
    want = torch.where(flat >= 0, segs[flat.clamp(min=0)] + rank_in, torch.full_like(flat, -1))
    assert torch.equal(route.dest_row.long(), want) and torch.equal(route.dest_rank >= 0, flat >= 0)
    x, go = (torch.randn(T, hid, device=dev).bfloat16() for _ in range(2))
    n, sent = int(segs[-1]), flat >= 0
    recv = ws.push(x, route, None)
    ref = torch.zeros(n, hid, dtype=torch.bfloat16, device=dev)
    ref[want[sent]] = x.repeat_interleave(k, 0)[sent]
    assert torch.equal(recv[:n], ref)                                                                     # the padding rows are zeros
    w = torch.rand(T, k, device=dev)
    y = torch.randn(recv.shape, device=dev).bfloat16()
    rows = torch.where(sent[:, None], y[want.clamp(min=0)].float(), torch.zeros((), device=dev)).view(T, k, hid)
    out, _ = ws.pull(y, route, w, False)
    torch.testing.assert_close(out.float(), (rows * w[..., None]).sum(1), rtol=2 ** -8, atol=k * 2 ** -9)
    d_y, d_w = ws.push_combine_grad(go, y, route, w)
    ref = torch.zeros(n, hid, device=dev)
    ref[want[sent]] = (go.float()[:, None] * w[..., None]).reshape(-1, hid)[sent]
    torch.testing.assert_close(d_y[:n].float(), ref, rtol=2 ** -8, atol=0)
    torch.testing.assert_close(d_w, (rows * go.float()[:, None]).sum(-1), rtol=1e-4, atol=1e-3)            # fp32 sums over `hid` products of size one
    torch.cuda.synchronize()
    fused_comm.check_status("one rank")


@pytest.mark.parametrize("T,k,E,hid,drop", [(1, 1, 3, 8, False), (300, 2, 4, 72, True), (0, 2, 4, 64, False)])
def test_one_rank_pull_with_the_gathered_rows(T, k, E, hid, drop):
    """The rows that a combine gathers, unweighted and in token order, zeros for dropped pairs; the sum is that of a pull without them."""
    from linear_moe_b200.ops import gemm
    from linear_moe_b200.parallel import fused_comm
    dev = torch.device("cuda", 0)
    torch.manual_seed(2)
    ws = fused_comm.MoeWorkspace(None, E, hid, T * k + gemm.ROW_ALIGN * E, dev)
    idx = torch.randint(-1 if drop else 0, E, (T, k), device=dev)
    route = ws.route(idx)
    y, w = torch.randn(ws.cap, hid, device=dev).bfloat16(), torch.rand(T, k, device=dev)
    out, rows = ws.pull(y, route, w, True)
    sent = (idx.reshape(-1) >= 0)[:, None]
    assert rows.shape == (T * k, hid) and torch.equal(rows, torch.where(sent, y[route.dest_row.clamp(min=0).long()], torch.zeros_like(rows)))
    assert torch.equal(out, ws.pull(y, route, w, False)[0])
    torch.cuda.synchronize()
    fused_comm.check_status("pull")


def test_one_rank_workspace_holds_no_buffers():
    """A workspace for many rows takes no device memory of its own on one rank, and a call with it leaves none behind."""
    from linear_moe_b200.ops.moe_fused import fused_moe
    from linear_moe_b200.parallel import fused_comm
    dev = torch.device("cuda", 0)
    T, k, E, hid, f = 64, 2, 4, 256, 64
    w1, w2 = torch.randn(E, hid, 2 * f, device=dev).bfloat16(), torch.randn(E, f, hid, device=dev).bfloat16()
    h, probs, idx = torch.randn(T, hid, device=dev).bfloat16(), torch.rand(T, k, device=dev), torch.randint(0, E, (T, k), device=dev)
    ws = fused_comm.MoeWorkspace(None, E, hid, 256 * E + T * k, dev)
    fused_moe(h, probs, idx, w1, w2, ws)                     # scratch and status words of the process
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    ws = fused_comm.MoeWorkspace(None, E, hid, 1 << 18, dev)
    out = fused_moe(h, probs, idx, w1, w2, ws)
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() - before <= out.numel() * 2 + 65536
