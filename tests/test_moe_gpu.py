"""MoE kernels and the expert-parallel layer against plain fp32 PyTorch references (single rank;
the multi-rank path runs in tests/mp_moe_worker.py when at least 2 GPUs are present)."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref_forward(x, gate, w13, w2, top_k, bias=None, idx=None):
    """fp32 reference. `idx` pins the expert choice (near-ties may flip between bf16 and fp32 logits)."""
    from fast_b200.models.moe import split_gate_up

    xf = x.float()
    logits = xf @ gate.float().t()
    if idx is None:
        sel = logits + (bias.float() if bias is not None else 0.0)
        idx = sel.topk(top_k, dim=-1).indices
    w = torch.softmax(logits.gather(1, idx), dim=-1)
    w1, w3 = split_gate_up(w13.float())
    out = torch.zeros_like(xf)
    for e in range(w13.shape[0]):
        tok, slot = (idx == e).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        h = xf[tok]
        a = torch.nn.functional.silu(h @ w1[e].t()) * (h @ w3[e].t())
        out = out.index_add(0, tok, (a @ w2[e].float().t()) * w[tok, slot].unsqueeze(1))
    return out, idx, w


def _rel(a, b):
    return ((a.float() - b.float()).abs().max() / (b.float().abs().max() + 1e-9)).item()


@pytest.mark.parametrize("E,K", [(8, 2), (256, 8), (64, 6)])
def test_route_topk_matches_torch(E, K):
    from fast_b200 import runtime

    C = runtime.ext()
    T = 1000
    g = torch.Generator(device="cuda").manual_seed(E)
    logits = torch.randn(T, E, generator=g, device="cuda")
    bias = torch.randn(E, generator=g, device="cuda") * 1.5
    nb = (T + C.ROUTE_TOKENS_PER_BLOCK - 1) // C.ROUTE_TOKENS_PER_BLOCK
    idx = torch.empty(T, K, dtype=torch.int32, device="cuda")
    w = torch.empty(T, K, dtype=torch.float32, device="cuda")
    slot = torch.zeros(nb * C.ROUTE_TOKENS_PER_BLOCK, K, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(nb, E, dtype=torch.int32, device="cuda")
    C.route_topk(logits, bias, K, idx, w, slot, cnt)
    ref_idx = (logits + bias).topk(K, dim=-1).indices
    assert torch.equal(idx.long(), ref_idx)
    ref_w = torch.softmax(logits.gather(1, ref_idx), dim=-1)
    assert torch.allclose(w, ref_w, atol=1e-5)
    # histogram and stable in-block ranks
    for b in range(nb):
        blk = idx[b * 128:(b + 1) * 128].reshape(-1).long()
        assert torch.equal(cnt[b].long(), torch.bincount(blk, minlength=E))
    flat = idx.reshape(-1).cpu()
    s = slot[:T].reshape(-1).cpu()
    seen = {}
    for i in range(min(flat.numel(), 128 * K)):
        e = int(flat[i])
        assert int(s[i]) == seen.get(e, 0)
        seen[e] = seen.get(e, 0) + 1


def test_route_topk_is_total_on_nan_inf_and_masked_rows():
    """Rows of NaN, of -inf, or with fewer than K selectable experts still get K distinct ids inside
    [0, E) and finite weights; rows with enough finite values route exactly like PyTorch."""
    from fast_b200 import runtime

    C = runtime.ext()
    T, E, K = 256, 64, 6
    g = torch.Generator(device="cuda").manual_seed(9)
    logits = torch.randn(T, E, generator=g, device="cuda")
    logits[0] = float("nan")
    logits[1] = float("-inf")
    logits[2, 3:] = float("-inf")            # three selectable experts, K = 6
    logits[3, ::2] = float("nan")            # half the experts unusable, still >= K finite
    logits[4, 5] = float("inf")
    idx = torch.empty(T, K, dtype=torch.int32, device="cuda")
    w = torch.empty(T, K, dtype=torch.float32, device="cuda")
    slot = torch.zeros(256, K, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(2, E, dtype=torch.int32, device="cuda")
    C.route_topk(logits, None, K, idx, w, slot, cnt)
    torch.cuda.synchronize()
    assert int(idx.min()) >= 0 and int(idx.max()) < E
    assert all(len(set(r)) == K for r in idx[:8].cpu().tolist())
    assert bool(torch.isfinite(w[[0, 1, 2, 3] + list(range(5, T))]).all())
    assert float(w[0].abs().sum()) == 0.0 and float(w[1].abs().sum()) == 0.0
    assert sorted(idx[2, :3].cpu().tolist()) == [0, 1, 2] and abs(float(w[2, :3].sum()) - 1.0) < 1e-5 and float(w[2, 3:].abs().sum()) == 0.0
    assert all(e % 2 == 1 for e in idx[3].cpu().tolist())
    ref = logits[5:].topk(K, dim=-1).indices
    assert torch.equal(idx[5:].long(), ref)
    assert int(cnt.sum()) == T * K


def test_expert_ids_out_of_range_are_skipped_and_reported():
    """Routing tables that name an expert outside [0, E) (a caller's own router gone wrong) are not
    used as indices: the entries are skipped, the status block names the site, the context lives."""
    from fast_b200 import runtime
    from fast_b200.models import MoELayer
    from fast_b200.parallel import Communicator

    comm = Communicator(heap_bytes=128 << 20, device=0)
    layer = MoELayer(comm, 256, 256, 4, 2, max_tokens=512, training=False)
    eng = layer.engine
    x = torch.randn(300, 256, device="cuda").to(torch.bfloat16)
    rs = eng.route((x @ layer.gate.t()).float())
    rs.topk_idx[7, 1] = 0x7FFFFFFF
    rs.topk_idx[9, 0] = -3
    eng.dispatch(x, rs)
    with pytest.raises(runtime.CollectiveTimeout) as e:
        comm.check()
    assert e.value.code == 2 and e.value.site == 11 and e.value.want == 4
    comm.reset()
    out = torch.empty(300, 256, dtype=torch.bfloat16, device="cuda")
    eng._C.combine_pull(comm.heap, eng.E, rs.topk_idx, rs.dest_row, rs.topk_w, eng._off(eng.y), eng._flag_off(1), 0, out, None, None, eng.H, eng.status,
                        eng.timeout_ns, 8, 0)
    with pytest.raises(runtime.CollectiveTimeout) as e:
        comm.check()
    assert e.value.site == 11
    assert int((torch.ones(8, device="cuda") * 3).sum().item()) == 24  # context still healthy


@pytest.mark.parametrize("T,H,E,K", [(300, 256, 8, 2), (1000, 512, 32, 6), (129, 1024, 4, 1)])
def test_fused_norm_router_forward_and_backward_match_torch(T, H, E, K):
    """RMSNorm + router logits + top-k (+ softmax-over-top-k weights) in one kernel, and its backward
    (gate, norm-weight and input gradients), against the same chain of plain fp32 PyTorch ops."""
    from fast_b200 import runtime

    C = runtime.ext()
    g = torch.Generator(device="cuda").manual_seed(T + E)
    h = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    nw = (1.0 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(torch.bfloat16)
    gate = (torch.randn(E, H, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    nb = (T + C.ROUTE_TOKENS_PER_BLOCK - 1) // C.ROUTE_TOKENS_PER_BLOCK
    hn = torch.empty_like(h)
    rstd = torch.empty(T, device="cuda")
    logits = torch.empty(T, E, device="cuda")
    idx = torch.empty(T, K, dtype=torch.int32, device="cuda")
    w = torch.empty(T, K, device="cuda")
    slot = torch.zeros(nb * C.ROUTE_TOKENS_PER_BLOCK, K, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(nb, E, dtype=torch.int32, device="cuda")
    eps = 1e-5
    C.norm_gate_route(h, nw, gate, None, K, eps, hn, rstd, logits, idx, w, slot, cnt)
    # fp32 reference with autograd; the expert choice is pinned to the kernel's (near-ties may flip)
    hr = h.float().requires_grad_()
    nwr = nw.float().requires_grad_()
    gr = gate.float().requires_grad_()
    hn_ref = hr * torch.rsqrt(hr.pow(2).mean(-1, keepdim=True) + eps) * nwr
    lg_ref = hn_ref @ gr.t()
    assert _rel(hn, hn_ref) < 1e-2 and _rel(logits, lg_ref) < 1e-2
    top_ref = lg_ref.topk(K, dim=-1)
    agree = (idx.long().sort(-1).values == top_ref.indices.sort(-1).values).all(-1).float().mean().item()
    assert agree > 0.98                                       # bf16 rounding of hn may flip near-ties
    assert int(idx.min()) >= 0 and int(idx.max()) < E and int(cnt.sum()) == T * K
    w_ref = torch.softmax(lg_ref.gather(1, idx.long()), dim=-1)
    assert torch.allclose(w, w_ref, atol=2e-2)
    for b in range(nb):
        blk = idx[b * 128:(b + 1) * 128].reshape(-1).long()
        assert torch.equal(cnt[b].long(), torch.bincount(blk, minlength=E))
    # backward: loss = sum(w * gw) + sum(hn * ghn)
    gw = torch.randn(T, K, generator=g, device="cuda")
    ghn = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    ((w_ref * gw).sum() + (hn_ref * ghn.float()).sum()).backward()
    grad_h = torch.empty_like(h)
    d_gate = torch.zeros(E, H, device="cuda")
    d_nw = torch.zeros(H, device="cuda")
    C.norm_gate_bwd(h, nw, gate, rstd, idx, w, gw, ghn, grad_h, d_gate, d_nw)
    assert _rel(grad_h, hr.grad) < 2e-2
    assert _rel(d_gate, gr.grad) < 2e-2
    assert _rel(d_nw, nwr.grad) < 2e-2


def test_elementwise_kernels():
    from fast_b200 import runtime
    from fast_b200.models.moe import split_gate_up

    C = runtime.ext()
    g = torch.Generator(device="cuda").manual_seed(1)
    rows, inter = 300, 384
    gu = torch.randn(rows, 2 * inter, generator=g, device="cuda").to(torch.bfloat16)
    act = torch.empty(rows, inter, device="cuda", dtype=torch.bfloat16)
    C.swiglu_fwd(gu, act)
    gt, ut = split_gate_up(gu.float().t().reshape(1, 2 * inter, rows))
    gt, ut = gt[0].t().requires_grad_(), ut[0].t().requires_grad_()
    ref = torch.nn.functional.silu(gt) * ut
    assert _rel(act, ref) < 1e-2
    dact = torch.randn(rows, inter, generator=g, device="cuda").to(torch.bfloat16)
    dgu = torch.empty_like(gu)
    C.swiglu_bwd(gu, dact, dgu, 0)
    ref.backward(dact.float())
    dg, du = split_gate_up(dgu.float().t().reshape(1, 2 * inter, rows))
    assert _rel(dg[0].t(), gt.grad) < 1e-2 and _rel(du[0].t(), ut.grad) < 1e-2
    # AdamW against torch.optim.AdamW on fp32
    p = torch.randn(4096, generator=g, device="cuda")
    grad = torch.randn(4096, generator=g, device="cuda").to(torch.bfloat16)
    pb = p.to(torch.bfloat16)
    master, m, v = pb.float().clone(), torch.zeros(4096, device="cuda"), torch.zeros(4096, device="cuda")
    ref_p = pb.float().clone().requires_grad_()
    opt = torch.optim.AdamW([ref_p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for step in (1, 2, 3):
        C.adamw(pb, master, m, v, grad, 1e-2, 0.9, 0.95, 1e-8, 0.1, step, 1.0)
        ref_p.grad = grad.float()
        opt.step()
    assert torch.allclose(master, ref_p.detach(), atol=1e-5, rtol=1e-5)
    assert torch.equal(pb, master.to(torch.bfloat16))


def test_adamw_of_several_tensors_is_the_single_update():
    """One launch over tensors of all kinds of lengths (less than a block's chunk, its multiples, one past; more tensors than one
    launch takes; different step numbers) gives the bits of one call per tensor."""
    from fast_b200 import runtime

    C = runtime.ext()
    g = torch.Generator(device="cuda").manual_seed(4)
    sizes = [8, 2040, 2048, 2056, 4096, 10000] * 3
    make = lambda: [torch.randn(n, generator=g, device="cuda") for n in sizes]
    grads = [x.to(torch.bfloat16) for x in make()]
    masters, ms, vs = make(), make(), [x.abs() for x in make()]
    steps = [1 + i % 5 for i in range(len(sizes))]
    clone = lambda ts: [t.clone() for t in ts]
    got = [[torch.empty_like(x) for x in grads], clone(masters), clone(ms), clone(vs)]
    want = [[torch.empty_like(x) for x in grads], clone(masters), clone(ms), clone(vs)]
    C.adamw_step(*got, grads, steps, 1e-2, 0.9, 0.95, 1e-8, 0.1, 0.5)
    for i in range(len(sizes)):
        C.adamw(want[0][i], want[1][i], want[2][i], want[3][i], grads[i], 1e-2, 0.9, 0.95, 1e-8, 0.1, steps[i], 0.5)
    assert all(torch.equal(a, b) for x, y in zip(got, want) for a, b in zip(x, y))


def test_quantise_rows_matches_a_torch_restatement():
    """Rows to e4m3 in 1 x 128 blocks: the scale is amax / 448 rounded up to a bf16 value, the bytes are
    round-to-nearest e4m3 of value / scale; value x scale comes back within e4m3's half-ulp."""
    from fast_b200 import runtime

    C = runtime.ext()
    g = torch.Generator(device="cuda").manual_seed(3)
    T, H = 77, 768
    x = (torch.randn(T, H, generator=g, device="cuda") * torch.logspace(-3, 2, T, device="cuda").unsqueeze(1)).to(torch.bfloat16)
    x[5, 128:256] = 0  # an all-zero block keeps a tiny positive scale
    q = torch.empty(T, H, dtype=torch.uint8, device="cuda")
    sc = torch.empty(T, H // 128, dtype=torch.float32, device="cuda")
    C.quantise_rows(x, q, sc, 8)
    blocks = x.float().reshape(T, H // 128, 128)
    want = blocks.abs().amax(-1).clamp_min(1e-12) / 448.0
    want = ((want.view(torch.int32) + 0xFFFF) & -65536).view(torch.float32)  # up to the next bf16 value
    assert torch.equal(sc, want)
    ref_q = (blocks / want.unsqueeze(-1)).to(torch.float8_e4m3fn)
    got = q.view(torch.float8_e4m3fn).reshape(T, H // 128, 128)
    # the kernel multiplies by a reciprocal: a value on a rounding boundary may land one code away
    assert (got.float() != ref_q.float()).float().mean().item() < 1e-3
    back = got.float() * sc.unsqueeze(-1)
    assert ((back - blocks).abs() <= blocks.abs().amax(-1, keepdim=True) * (1.0 / 14) + 1e-12).all()
    assert torch.count_nonzero(back[5, 1]) == 0


def test_embedding_index_is_a_stable_sort_by_id():
    """The counting sort that feeds the embedding gradient equals torch's stable sort, with few and with heavy duplicates."""
    from fast_b200 import runtime

    C = runtime.ext()
    g = torch.Generator(device="cuda").manual_seed(11)
    for T, V, hot in ((5000, 3000, 0), (4097, 70000, 0), (3000, 50, 0), (2500, 1000, 2000)):
        ids = torch.randint(0, V, (T,), generator=g, device="cuda")
        if hot:
            ids[torch.randperm(T, generator=g, device="cuda")[:hot]] = 7     # one id taking most of the positions
        sid, perm = C.embedding_index(ids, V)
        rs, rp = torch.sort(ids, stable=True)
        assert torch.equal(sid, rs) and torch.equal(perm, rp)


@pytest.mark.parametrize("T,V,H,spread", [(1, 7, 256, 7), (33, 50, 264, 50), (300, 40, 256, 3), (4096, 1000, 256, 1000), (4097, 40000, 256, 40000), (5000, 33, 512, 2)])
def test_embedding_gradient_of_any_length(T, V, H, spread):
    """Pairwise search (up to 4096 tokens) and counting sort, rare and heavy duplicates: position-order fp32 sums, zeros elsewhere."""
    from fast_b200.ops import fused

    g = torch.Generator(device="cuda").manual_seed(T)
    ids = torch.randint(0, spread, (T,), generator=g, device="cuda") * (V // spread)
    table = torch.randn(V, H, generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    go = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    table.grad = None
    fused.embedding(ids, table).backward(go)
    want = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids, go.double())
    assert _rel(table.grad, want.float()) < 1e-2
    assert bool((table.grad[torch.bincount(ids, minlength=V) == 0] == 0).all())


@pytest.mark.parametrize("T,V,H,step", [(0, 40, 64, 1), (4096, 513, 520, 512), (4096, 2200000, 8, 2097152), (300, 32769, 2048, 1024), (4095, 9000, 1032, 512), (257, 32000, 4096, 31999)])
def test_embedding_gradient_of_few_positions_in_one_block(T, V, H, step):
    """Ids that all fall to one block's rows, rows that share a bit of its filter (2097152 apart), ids outside the table, ragged
    widths. n fp32 additions of bf16 values, one rounding to bf16: an error of at most 2^-8 of the sum plus n 2^-24 of the terms."""
    from fast_b200 import _C

    g = torch.Generator(device="cuda").manual_seed(T + V)
    ids = torch.randint(0, (V - 1) // step + 1, (T,), generator=g, device="cuda") * step
    if T:
        ids[::5], ids[3::7] = V, -1
    go = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    got = _C.embedding_grad(ids, V, go)
    used = (ids >= 0) & (ids < V)
    want = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids[used], go[used].double())
    terms = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids[used], go[used].double().abs())
    n = torch.bincount(ids[used], minlength=V).double()[:, None]
    assert bool(((got.double() - want).abs() <= 2.0**-8 * want.abs() + n * 2.0**-24 * terms + 1e-30).all())
    assert bool((got[n[:, 0] == 0] == 0).all())


@pytest.mark.parametrize("V,H", [(9, 264), (16, 2056), (8193, 8)])
def test_embedding_gradient_of_many_positions_with_frequent_ids(V, H):
    """Rows of 0, 1, 16 (one warp), 17, 24 and thousands of positions (the block's warps together), the last row of a table that is
    no multiple of eight rows among them. n fp32 additions of bf16 values, one rounding to bf16."""
    from fast_b200 import _C

    rows = [(0, 1), (1, 16), (2, 17), (4, 24), (5, 1700), (V - 1, 3000)]
    ids = torch.cat([torch.full((n,), v) for v, n in rows])
    g = torch.Generator().manual_seed(V)
    ids = ids[torch.randperm(ids.numel(), generator=g)].cuda()
    go = torch.randn(ids.numel(), H, generator=g).to(torch.bfloat16).cuda()
    got = _C.embedding_grad(ids, V, go)
    want = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids, go.double())
    terms = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids, go.double().abs())
    n = torch.bincount(ids, minlength=V).double()[:, None]
    assert ids.numel() > 4096 and bool(((got.double() - want).abs() <= 2.0**-8 * want.abs() + n * 2.0**-24 * terms).all())


@pytest.mark.parametrize("T,H,I,E,K", [(1, 256, 256, 4, 2), (127, 512, 256, 8, 2), (130, 1024, 256, 12, 3), (700, 2048, 256, 8, 2)])
def test_loss_inside_the_layer_matches_the_separate_ops(T, H, I, E, K):
    """mean((h + MoE(RMSNorm(h)))^2) with loss and gradients made inside combine, the backward dispatch and the norm's backward,
    against the same layer followed by the separate residual loss. Twice: tickets are clean for the next step."""
    from fast_b200.models import MoELayer
    from fast_b200.ops import fused
    from fast_b200.parallel import Communicator

    comm = Communicator(heap_bytes=256 << 20, device=0)
    layer = MoELayer(comm, H, I, E, K, max_tokens=T)
    assert layer.engine.can_fuse_gate()
    g = torch.Generator(device="cuda").manual_seed(T)
    nw = (1.0 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(torch.bfloat16).requires_grad_()
    for _ in range(2):
        h0 = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
        got = []
        for inside in (True, False):
            h = h0.clone().requires_grad_()
            for p in (nw, layer.gate, layer.w13, layer.w2):
                p.grad = None
            loss = layer.mean_square_from_residual(h, nw, 1e-5) if inside else fused.residual_mean_square(h, layer.forward_from_residual(h, nw, 1e-5))
            (loss * 3.0).backward()
            comm.check()
            got.append([loss.detach(), h.grad, nw.grad, layer.gate.grad, layer.w13.grad, layer.w2.grad])
        for a, b in zip(*got):
            assert _rel(a, b) < 2e-2


def test_fused_embedding_and_loss_match_torch():
    from fast_b200.ops import fused

    g = torch.Generator(device="cuda").manual_seed(5)
    table = (torch.randn(300, 256, generator=g, device="cuda") * 0.1).to(torch.bfloat16).requires_grad_()
    ids = torch.randint(0, 300, (4, 500), generator=g, device="cuda")
    other = (torch.randn(2000, 256, generator=g, device="cuda") * 0.1).to(torch.bfloat16).requires_grad_()
    loss = fused.residual_mean_square(fused.embedding(ids.reshape(-1), table), other)
    loss.backward()
    t2 = table.detach().clone().requires_grad_()
    o2 = other.detach().clone().requires_grad_()
    ref = (torch.nn.functional.embedding(ids.reshape(-1), t2) + o2).float().pow(2).mean()
    ref.backward()
    assert abs(loss.item() - ref.item()) < 1e-3 * abs(ref.item())
    assert _rel(other.grad, o2.grad) < 2e-2
    assert _rel(table.grad, t2.grad) < 2e-2


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("E,K,H,I,T,fp8", [(4, 2, 256, 256, 300, False), (8, 2, 512, 384, 1000, False), (32, 8, 256, 128, 513, False), (8, 2, 256, 256, 300, True),
                                           (8, 2, 256, 256, 300, "direct")])
def test_moe_forward_single_rank(E, K, H, I, T, fp8, overlap):
    from fast_b200.models import MoELayer
    from fast_b200.parallel import Communicator

    comm = Communicator(heap_bytes=256 << 20, device=0)
    layer = MoELayer(comm, H, I, E, K, max_tokens=1024, fp8_dispatch=bool(fp8), training=False, router_bias=True, overlap_dispatch=overlap,
                     fp8_direct=fp8 == "direct")
    layer.eval()
    g = torch.Generator(device="cuda").manual_seed(7)
    layer.router_bias.data = torch.randn(E, generator=g, device="cuda") * 0.5
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        out = layer(x)
        out2 = layer(x)  # second call: epochs, counters and pads must be reusable
    comm.check()
    ref, _, _ = _ref_forward(x, layer.gate, layer.w13, layer.w2, K, layer.router_bias, idx=layer.last_route.topk_idx.long())
    tol = 6e-2 if fp8 else 2e-2
    assert _rel(out, ref) < tol
    assert torch.equal(out, out2)
    tm = layer.engine.traffic_matrix()
    assert int(tm.sum().item()) == T * K


@pytest.mark.parametrize("E,K,H,I,T,fp8", [(8, 2, 512, 384, 1, False), (5, 3, 768, 256, 7, False), (32, 8, 256, 128, 128, False), (256, 8, 256, 128, 33, False),
                                            (8, 2, 512, 384, 64, True), (8, 2, 512, 384, 129, False), (40, 4, 7168, 256, 2, True)])
def test_forward_layer_of_few_tokens(E, K, H, I, T, fp8):
    """The routes a decode step takes: logits, choice, ranks and split scan in one kernel (up to 128 tokens), rows shared by
    the warps of a block, narrow GEMM tiles with cut reductions. Three steps in a row on other tokens; the routing tables
    agree with each other and the output with fp32."""
    from fast_b200.models import MoELayer
    from fast_b200.parallel import Communicator

    comm = Communicator(heap_bytes=256 << 20, device=0)
    layer = MoELayer(comm, H, I, E, K, max_tokens=max(T, 200), fp8_dispatch=fp8, router_bias=True, training=False).eval()
    g = torch.Generator(device="cuda").manual_seed(T)
    layer.router_bias.data.copy_(torch.randn(E, generator=g, device="cuda") * 0.5)
    for n in (T, max(1, T - 1), T):
        x = torch.randn(n, H, generator=g, device="cuda").to(torch.bfloat16)
        with torch.no_grad():
            y = layer(x)
        comm.check()
        rs, eng = layer.last_route, layer.engine
        idx = rs.topk_idx.long()
        want, _, w = _ref_forward(x, layer.gate, layer.w13, layer.w2, K, idx=idx)
        assert _rel(y, want) < (8e-2 if fp8 else 2e-2)
        sel = (x @ layer.gate.t()).float() + layer.router_bias
        top = sel.topk(K, dim=-1)
        assert bool((sel.gather(1, idx) >= top.values[:, -1:] - 2e-2).all()) and all(len(set(r)) == K for r in idx.tolist())
        assert torch.allclose(rs.topk_w, w, atol=2e-2)
        counts = torch.bincount(idx.reshape(-1), minlength=E)
        assert torch.equal(rs.group_rows.long(), counts) and int(eng.traffic_matrix()[0, 0]) == n * K
        off = torch.cat([torch.zeros(1, dtype=torch.long, device="cuda"), torch.cumsum((counts + 255) // 256 * 256, 0)])
        assert torch.equal(rs.group_off.long(), off)
        rows = rs.dest_row.long()
        assert bool(((rows >= off[idx]) & (rows < off[idx] + counts[idx])).all()) and rows.unique().numel() == n * K


@pytest.mark.parametrize("H,in_kernel", [(57344, True), (57600, False), (65536, False)])
def test_few_tokens_of_the_widest_rows(H, in_kernel):
    """A row that the routing kernel's shared memory cannot hold is routed through the GEMM: a layer of any width takes few tokens."""
    from fast_b200.models import MoELayer
    from fast_b200.parallel import Communicator

    comm = Communicator(heap_bytes=512 << 20, device=0)
    layer = MoELayer(comm, H, 256, 2, 1, max_tokens=4, training=False, init_std=0.01).eval()
    x = torch.randn(3, H, generator=torch.Generator(device="cuda").manual_seed(H), device="cuda").to(torch.bfloat16)
    assert layer.engine._gate_in_kernel(x, layer.gate) == in_kernel
    with torch.no_grad():
        y = layer(x)
    comm.check()
    want, _, _ = _ref_forward(x, layer.gate, layer.w13, layer.w2, 1, idx=layer.last_route.topk_idx.long())
    assert _rel(y, want) < 2e-2
    comm.close()


@pytest.mark.parametrize("fp8,overlap", [(False, False), (True, False), (False, True), (True, True)])
def test_forward_layer_without_tokens(fp8, overlap):
    """A step of no tokens returns no rows, and the step after it is as if it had not been."""
    from fast_b200.models import MoELayer
    from fast_b200.parallel import Communicator

    comm = Communicator(heap_bytes=128 << 20, device=0)
    layer = MoELayer(comm, 256, 256, 8, 2, max_tokens=512, fp8_dispatch=fp8, training=False, overlap_dispatch=overlap).eval()
    x = torch.randn(300, 256, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        want = layer(x)
        assert layer(x[:0]).shape == (0, 256) and int(layer.engine.traffic_matrix().sum()) == 0
        got = layer(x)
    comm.check()
    assert torch.equal(got, want)


@pytest.mark.parametrize("fused", [False, True])
def test_training_layer_without_tokens(fused):
    """Forward and backward of no tokens: every parameter's gradient is zero, the input's has no rows."""
    from fast_b200.models import MoELayer
    from fast_b200.parallel import Communicator

    comm = Communicator(heap_bytes=128 << 20, device=0)
    layer = MoELayer(comm, 256, 256, 8, 2, max_tokens=512)
    norm = torch.ones(256, dtype=torch.bfloat16, device="cuda", requires_grad=True)
    x = torch.empty(0, 256, dtype=torch.bfloat16, device="cuda", requires_grad=True)
    out = layer.forward_from_residual(x, norm, 1e-5) if fused else layer(x)
    assert out.shape == x.shape
    out.sum().backward()
    comm.check()
    assert x.grad.shape == x.shape
    for p in (layer.gate, layer.w13, layer.w2) + ((norm,) if fused else ()):
        assert int(p.grad.count_nonzero()) == 0


def _two_ranks_words(C, flags=4):
    """Heaps of two ranks in this process, and where `flags` words per rank lie in both."""
    heaps = C.SymmHeap.create_local_group(2, 1 << 20, 0)
    off = [h.alloc(64 * 8) for h in heaps][0]
    return heaps, off, [h.tensor(off, [flags], torch.int64) for h in heaps]


@pytest.mark.parametrize("epoch_on_device", [False, True])
def test_rank_without_tokens_says_that_its_rows_are_final(epoch_on_device):
    """Combine of a rank without tokens writes its ready flag on every rank (their tokens may have gone to its experts). The
    peer's flag is there before the launch, so nothing waits."""
    from fast_b200 import runtime

    C = runtime.ext()
    heaps, off, flags = _two_ranks_words(C)
    st = C.StatusBlock()
    flags[0][1] = 7
    none = torch.empty(0, 2, dtype=torch.int32, device="cuda")
    epoch = torch.full((1,), 7, dtype=torch.int64, device="cuda")
    out = torch.empty(0, 256, dtype=torch.bfloat16, device="cuda")
    C.combine_pull(heaps[0], 2, none, none, none.float(), 0, off, 0 if epoch_on_device else 7, out, None, None, 256, st, int(1e9), 8,
                   epoch.data_ptr() if epoch_on_device else 0, True)
    assert st.read()[0] == 0
    assert flags[1].tolist() == [7, 0, 0, 0] and flags[0].tolist() == [7, 7, 0, 0]


def test_rank_without_tokens_joins_the_entry_handshake():
    """The backward dispatch of a rank without tokens publishes that its receive buffers may be written."""
    from fast_b200 import runtime

    C = runtime.ext()
    heaps, off, flags = _two_ranks_words(C)
    st = C.StatusBlock()
    flags[0][1] = 7
    none = torch.empty(0, 2, dtype=torch.int32, device="cuda")
    x = torch.empty(0, 256, dtype=torch.bfloat16, device="cuda")
    send_base = torch.zeros(2, dtype=torch.int32, device="cuda")
    C.dispatch_push(heaps[0], x, none, none.float(), none, none, send_base, none, False, False, 0, 0, -1, off, 7, st, int(1e9), 8, None, 0, 0,
                    None, None, None, none.float(), 0)
    assert st.read()[0] == 0
    assert flags[1].tolist() == [7, 0, 0, 0] and flags[0].tolist() == [7, 7, 0, 0]


def test_views_that_start_between_16_byte_words():
    """A router gate may be a view at any element (few tokens: the routing kernel's 16-byte reads give way to the GEMM); rows, which
    every kernel of the chain reads in 16-byte words, are refused on the host."""
    from fast_b200.models import MoELayer
    from fast_b200.ops import fused
    from fast_b200.parallel import Communicator

    comm = Communicator(heap_bytes=128 << 20, device=0)
    layer = MoELayer(comm, 256, 256, 8, 2, max_tokens=512, training=False).eval()
    x = torch.randn(5, 256, device="cuda").to(torch.bfloat16)

    def moved(t):
        return torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view_as(t).copy_(t.detach())

    with torch.no_grad():
        layer(x)
        want = layer.last_route.topk_idx.clone()
        layer.gate.data = moved(layer.gate)
        y = layer(x)
        assert bool((layer.last_route.topk_idx == want).float().mean() > 0.9)   # the two sums round some logits differently
        ref, _, _ = _ref_forward(x, layer.gate, layer.w13, layer.w2, 2, idx=layer.last_route.topk_idx.long())
        assert _rel(y, ref) < 2e-2
        with pytest.raises(RuntimeError, match="16 bytes"):
            layer(moved(x))
    with pytest.raises(RuntimeError, match="16 bytes"):
        fused.residual_mean_square(x, moved(x))
    comm.check()


def test_weights_written_after_dispatch_are_waited_for(monkeypatch):
    """The expert GEMM may read its weights before the kernel ahead of it has ended only where its caller says that this kernel does
    not write them: the layer does, a caller of the engine's own steps does not by default."""
    from fast_b200.models import MoELayer
    from fast_b200.ops import gemm
    from fast_b200.parallel import Communicator

    if not gemm.USE_PAIR:
        pytest.skip("one-CTA kernels are not launched early")
    comm = Communicator(heap_bytes=128 << 20, device=0)
    layer = MoELayer(comm, 256, 256, 8, 2, max_tokens=512, training=False).eval()
    eng, early, fwd = layer.engine, [], gemm.grouped_gemm_fwd
    monkeypatch.setattr(gemm, "grouped_gemm_fwd", lambda *a, **k: (early.append(k["scratch"].early), fwd(*a, **k))[1])
    x = torch.randn(300, 256, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        want = layer(x)
        assert early == [True, True]
        early.clear()
        w13 = torch.zeros_like(layer.w13)
        rs = eng.route_gate(x, layer.gate)
        eng.dispatch(x, rs)
        w13.copy_(layer.w13)
        eng.experts_forward(w13, layer.w2, rs)
        assert early == [False, True]
        assert torch.equal(eng.combine(rs, rs.topk_w), want)
    comm.check()


@pytest.mark.parametrize("T", [5, 300])
@pytest.mark.parametrize("fp8", [False, True])
def test_layer_alone_takes_its_engine_s_steps(T, fp8):
    """A rank that is alone has shorter launch calls of its own. They give the bits of the general ones, they follow a grid that is set
    after construction, and a step that is replaced is the one that runs."""
    from fast_b200.models import MoELayer
    from fast_b200.ops import gemm
    from fast_b200.parallel import Communicator

    if not gemm.USE_PAIR:
        pytest.skip("the one-CTA kernels have the general launches only")
    comm = Communicator(heap_bytes=128 << 20, device=0)
    layer = MoELayer(comm, 256, 256, 8, 2, max_tokens=512, fp8_dispatch=fp8, training=False, router_bias=True).eval()
    eng, local = layer.engine, layer.engine._local
    assert local is not None
    x = torch.randn(T, 256, generator=torch.Generator(device="cuda").manual_seed(T), device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        want, rows = layer(x), layer.last_route.dest_row.clone()
        unweighted = eng.combine(layer.last_route, None)
        eng._local = None
        assert torch.equal(layer(x), want) and torch.equal(layer.last_route.dest_row, rows)
        assert torch.equal(eng.combine(layer.last_route, None), unweighted)
        eng._local = local
        grid, seen, dispatch = eng.comm_ctas, [], eng.dispatch
        eng.comm_ctas = 3
        assert torch.equal(layer(x), want)
        eng.comm_ctas = 0                                     # refused on the host
        with pytest.raises(RuntimeError):
            eng.dispatch(x, layer.last_route)
        with pytest.raises(RuntimeError):
            eng.combine(layer.last_route, layer.last_route.topk_w)
        eng.comm_ctas = grid
        eng.dispatch = lambda rows_in, rs: (seen.append(rows_in.shape[0]), dispatch(rows_in, rs))[1]
        assert torch.equal(layer(x), want) and seen == [T]
    comm.check()


def test_forward_layer_in_cuda_graph():
    """The forward-only layer captured in a CUDA graph replays correctly on new inputs (the step's
    epoch lives in device memory, so a replay is a new step)."""
    from fast_b200.models import MoELayer
    from fast_b200.parallel import Communicator

    E, K, H, I, T = 8, 2, 256, 256, 384
    comm = Communicator(heap_bytes=256 << 20, device=0)
    layer = MoELayer(comm, H, I, E, K, max_tokens=512, training=False, graph_mode=True)
    layer.eval()
    layer.capture(T)
    g = torch.Generator(device="cuda").manual_seed(21)
    for it in range(3):
        x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
        out = layer.forward_graphed(x).clone()
        comm.check()
        ref, _, _ = _ref_forward(x, layer.gate, layer.w13, layer.w2, K, idx=layer.last_route.topk_idx[:T].long())
        assert _rel(out, ref) < 2e-2, f"replay {it}"
    assert int(layer.engine.epoch_dev.item()) == 2 + 3  # two warm-up steps + three replays


def test_receive_capacity_guard_refuses_step():
    """A step that needs more receive rows than the buffers hold is refused on the device
    (no row is written out of bounds) and reported through the status block."""
    from fast_b200 import runtime
    from fast_b200.models import MoELayer
    from fast_b200.parallel import Communicator

    comm = Communicator(heap_bytes=128 << 20, device=0)
    layer = MoELayer(comm, 256, 256, 4, 2, max_tokens=1024, training=False, capacity_rows=512)
    layer.eval()
    x = torch.randn(900, 256, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        layer(x)  # needs ~1800 rows (+ padding) > 512
    with pytest.raises(runtime.CollectiveTimeout) as e:
        comm.check()
    assert e.value.site == 10 and e.value.want == 512 and e.value.seen > 512
    assert int((torch.ones(8, device="cuda") * 3).sum().item()) == 24  # context still healthy


def test_moe_backward_single_rank():
    from fast_b200.models import MoELayer
    from fast_b200.parallel import Communicator

    E, K, H, I, T = 8, 2, 256, 256, 600
    comm = Communicator(heap_bytes=256 << 20, device=0)
    layer = MoELayer(comm, H, I, E, K, max_tokens=1024)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    gout = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    out = layer(x)
    out.backward(gout)
    comm.check()
    # fp32 reference with autograd
    xr = x.detach().float().requires_grad_()
    gate = layer.gate.detach().float().requires_grad_()
    w13 = layer.w13.detach().float().requires_grad_()
    w2 = layer.w2.detach().float().requires_grad_()
    ref, _, _ = _ref_forward(xr, gate, w13, w2, K, idx=layer.last_route.topk_idx.long())
    ref.backward(gout.float())
    assert _rel(out, ref) < 2e-2
    assert _rel(x.grad, xr.grad) < 3e-2
    assert _rel(layer.w13.grad, w13.grad) < 3e-2
    assert _rel(layer.w2.grad, w2.grad) < 3e-2
    assert _rel(layer.gate.grad, gate.grad) < 5e-2


def test_block_model_trains():
    from fast_b200.models import MixtralBlockModel
    from fast_b200.parallel import Communicator
    from fast_b200.utils import FusedAdamW

    comm = Communicator(heap_bytes=256 << 20, device=0)
    model = MixtralBlockModel(comm, vocab=512, hidden=256, inter=256, num_experts=4, top_k=2, max_tokens=512)
    opt = FusedAdamW(model.expert_parameters(), lr=5e-3)
    ids = torch.randint(0, 512, (2, 256), device="cuda", generator=torch.Generator(device="cuda").manual_seed(0))
    losses = []
    for _ in range(5):
        opt.zero_grad()
        loss = model(ids)
        loss.backward()
        opt.step()
        losses.append(float(loss.item()))
    comm.check()
    assert all(l == l for l in losses) and losses[-1] < losses[0]


def test_optimizer_in_backward_matches_late_step():
    """Applying W2's AdamW update inside the backward pass (side stream) gives bit-identical weights."""
    from fast_b200.models import MixtralBlockModel
    from fast_b200.parallel import Communicator
    from fast_b200.utils import FusedAdamW

    ids = torch.randint(0, 512, (2, 256), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    results = []
    for early in (False, True):
        comm = Communicator(heap_bytes=256 << 20, device=0)
        model = MixtralBlockModel(comm, vocab=512, hidden=256, inter=256, num_experts=4, top_k=2, max_tokens=512, seed=3)
        opt = FusedAdamW(model.expert_parameters(), lr=1e-2)
        if early:
            model.moe.attach_optimizer(opt)
        for _ in range(3):
            opt.zero_grad()
            model(ids).backward()
            opt.step()
        comm.check()
        torch.cuda.synchronize()
        results.append((model.moe.w13.detach().clone(), model.moe.w2.detach().clone()))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    assert not torch.equal(results[0][1], torch.zeros_like(results[0][1]))


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs 2 GPUs")
def test_moe_multi_process():
    n = min(torch.cuda.device_count(), 8)
    env = dict(os.environ, NCCL_NVLS_ENABLE="0")
    r = subprocess.run([sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={n}", "--master-addr", "127.0.0.1",
                        "--master-port", "29543", os.path.join(os.path.dirname(__file__), "mp_moe_worker.py")], capture_output=True, text=True, env=env, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "MOE_MP_OK" in r.stdout


@pytest.mark.parametrize("T,E,K,H", [(1, 8, 2, 256), (1, 64, 8, 512), (2, 8, 8, 1024), (17, 5, 3, 256), (33, 33, 4, 512), (128, 32, 8, 768), (127, 256, 2, 256)])
@pytest.mark.parametrize("capacity", [None, 256])
def test_routing_of_few_tokens_alone(T, E, K, H, capacity):
    """The kernel that makes logits, choice, ranks and the split scan of few tokens: choice and weights against torch, ranks, rows and
    groups against a count in token order; a step whose padded rows exceed the capacity is refused, with empty groups."""
    from fast_b200.parallel import Communicator
    from fast_b200.parallel.ep import ExpertParallel
    from fast_b200.ops import gemm

    comm = Communicator(heap_bytes=256 << 20, device=0)
    eng = ExpertParallel(comm, E, H, 256, K, max_tokens=128, training=False, capacity_rows=capacity)
    g = torch.Generator(device="cuda").manual_seed(T * 131 + E)
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    gate = (torch.randn(E, H, generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    assert eng._gate_in_kernel(x, gate)
    before = eng.arrive_target.clone()
    rs = eng.route_gate(x, gate)
    torch.cuda.synchronize()
    logits = (x.float() @ gate.float().t()).to(torch.bfloat16).float()
    idx = rs.topk_idx.long()
    chosen = logits.gather(1, idx)
    # a choice is right if nothing that was left out is larger by more than a rounding of a bf16 logit
    left = logits.scatter(1, idx, float("-inf")).max(1).values if K < E else torch.full((T,), float("-inf"), device="cuda")
    assert bool((chosen.min(1).values >= left - logits.abs().max() * 2 ** -7).all()) and bool((idx.sort(1).values.diff(dim=1) > 0).all())
    assert torch.allclose(rs.topk_w, torch.softmax(chosen, 1), atol=2e-2)   # two bf16 logits off by one rounding: exp(2 * 2^-8) - 1
    counts = torch.bincount(idx.flatten(), minlength=E)
    align = gemm.row_align()
    padded = (counts + align - 1) // align * align
    if int(padded.sum()) > eng.cap:
        with pytest.raises(Exception):
            comm.check()
        comm.status.clear()
        assert int(rs.group_rows.abs().sum()) == 0 and int(rs.group_off.abs().sum()) == 0
        return
    comm.check()
    assert torch.equal(rs.group_rows.long(), counts) and torch.equal(rs.group_off.long(), torch.cat([padded.new_zeros(1), padded.cumsum(0)]))
    assert torch.equal((eng.arrive_target - before)[0], counts) and int(eng.traffic[0, 0]) == T * K
    assert torch.equal(rs.send_base.long(), rs.group_off[:E].long())
    seen = [0] * E
    slots = rs.slot_in_block[:T].tolist()
    for t, row in enumerate(idx.tolist()):
        for j, e in enumerate(row):
            assert slots[t][j] == seen[e]
            seen[e] += 1


@pytest.mark.parametrize("T,E,H", [(1, 8, 12032), (2, 8, 12032), (2, 8, 12288), (1, 256, 11776), (2, 256, 12032)])
def test_routing_of_few_tokens_in_rows_that_nearly_fill_the_unasked_shared_memory(T, E, H):
    """4 H bytes for a token's row, 32 words or one per expert, and a kilobyte of static tables: just below and above the 48 KiB that a launch may use unasked."""
    test_routing_of_few_tokens_alone(T, E, 2, H, 1024)
