"""tcgen05 grouped GEMM against a plain PyTorch fp32 reference of the same contraction."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["one_cta", "cta_pair"], autouse=True)
def kernel_variant(request):
    """Every case runs on the one-CTA kernel and on the CTA-pair (cta_group::2) kernel."""
    from fast_b200.ops import gemm

    old = gemm.USE_PAIR
    gemm.USE_PAIR = request.param == "cta_pair"
    yield request.param
    gemm.USE_PAIR = old


def _setup(G, N, K, counts, seed=0):
    from fast_b200.ops import pad_group_offsets

    g = torch.Generator(device="cuda").manual_seed(seed)
    counts = torch.tensor(counts, device="cuda")
    off = pad_group_offsets(counts)
    R = int(off[-1].item())
    a = torch.zeros(R, K, device="cuda", dtype=torch.bfloat16)
    for i in range(G):
        s, c = int(off[i]), int(counts[i])
        a[s:s + c] = torch.randn(c, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(G, N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    return counts, off, R, a, w


def _close(got, want, tol=2e-2):
    if want.numel() == 0:
        return
    err = (got.float() - want).abs().max().item()
    scale = want.abs().max().item() + 1e-6
    assert err / scale < tol, f"max err {err} vs scale {scale}"


@pytest.mark.parametrize("G,N,K,counts", [(1, 256, 64, [128]), (1, 256, 256, [128]), (2, 512, 320, [200, 77]), (4, 768, 512, [0, 300, 128, 1])])
def test_forward(G, N, K, counts):
    from fast_b200.ops import gemm

    counts, off, R, a, w = _setup(G, N, K, counts)
    out = torch.full((R, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_fwd(a, w, off, out)
    gemm.check()
    for i in range(G):
        s, e = int(off[i]), int(off[i + 1])
        _close(out[s:e], a[s:e].float() @ w[i].float().T)


def test_other_views_at_the_same_address():
    """Calls on memory that an earlier call used in another way: refused views stay refused, other pitches are followed."""
    from fast_b200.ops import gemm

    G, N, K = 1, 256, 256
    counts, off, R, a, w = _setup(G, N, K, [200], seed=8)
    want = a.float() @ w[0].float().T
    out = torch.empty(R, N, device="cuda", dtype=torch.bfloat16)
    for _ in range(2):
        gemm.grouped_gemm_fwd(a, w, off, out)
        _close(out[:200], want[:200])
        for bad in (w.transpose(1, 2), w.view(torch.float16)):
            with pytest.raises((RuntimeError, AssertionError)):
                gemm.grouped_gemm_fwd(a, bad, off, out)
    act, buf = torch.empty(R, N // 2, device="cuda", dtype=torch.bfloat16), torch.empty(R, 2 * N, device="cuda", dtype=torch.bfloat16)
    for gate_up in (buf[:, :N], buf.view(-1)[: R * N].view(R, N), buf[:, :N]):
        gate_up.fill_(float("nan"))
        gemm.grouped_gemm_fwd(a, w, off, act, swiglu=True, gate_up_out=gate_up)
        _close(gate_up[:200], want[:200])
    gemm.check()


def test_forward_swiglu():
    from fast_b200.ops import gemm

    G, N, K = 2, 512, 256
    counts, off, R, a, w = _setup(G, N, K, [130, 256], seed=3)
    act = torch.empty(R, N // 2, device="cuda", dtype=torch.bfloat16)
    gu = torch.empty(R, N, device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_fwd(a, w, off, act, swiglu=True, gate_up_out=gu)
    gemm.check()
    for i in range(G):
        s, e = int(off[i]), int(off[i + 1])
        full = a[s:e].float() @ w[i].float().T
        _close(gu[s:e], full)
        t = full.view(e - s, N // 256, 2, 128)
        _close(act[s:e], (torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(e - s, N // 2))


@pytest.mark.parametrize("G,N,K,counts", [(1, 64, 256, [128]), (2, 320, 512, [200, 77]), (3, 512, 768, [1, 0, 257])])
def test_dgrad(G, N, K, counts):
    from fast_b200.ops import gemm

    counts, off, R, dy, w = _setup(G, K, N, counts, seed=5)  # dy [R, N]; w [G, N, K]
    w = w.transpose(1, 2).contiguous()  # [G, N, K]
    out = torch.full((R, K), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_dgrad(dy, w, off, out)
    gemm.check()
    for i in range(G):
        s, e = int(off[i]), int(off[i + 1])
        _close(out[s:e], dy[s:e].float() @ w[i].float())


@pytest.mark.parametrize("G,N,K,counts", [(1, 256, 256, [128]), (2, 256, 512, [200, 77]), (3, 512, 256, [1, 0, 257])])
def test_wgrad(G, N, K, counts):
    from fast_b200.ops import gemm

    counts, off, R, x, _ = _setup(G, 256, K, counts, seed=7)
    g = torch.Generator(device="cuda").manual_seed(11)
    dy = torch.zeros(R, N, device="cuda", dtype=torch.bfloat16)
    for i in range(G):
        s, c = int(off[i]), int(counts[i])
        dy[s:s + c] = torch.randn(c, N, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((G, N, K), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_wgrad(dy, x, off, out)
    gemm.check()
    for i in range(G):
        s, e = int(off[i]), int(off[i + 1])
        _close(out[i], dy[s:e].float().T @ x[s:e].float())


def test_large_shape_matches():
    from fast_b200.ops import gemm

    G, N, K = 2, 2048, 1024
    counts, off, R, a, w = _setup(G, N, K, [1500, 900], seed=9)
    out = torch.empty(R, N, device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_fwd(a, w, off, out)
    gemm.check()
    for i in range(G):
        s, e = int(off[i]), int(off[i + 1])
        _close(out[s:e], a[s:e].float() @ w[i].float().T)


def test_dgrad_with_fused_swiglu_backward(kernel_variant):
    """dgrad of the second projection with the SwiGLU backward applied in its epilogue."""
    if kernel_variant != "cta_pair":
        pytest.skip("only the CTA-pair kernel carries this epilogue")
    from fast_b200.ops import gemm

    G, H, I = 2, 256, 512
    counts, off, R, dy, _ = _setup(G, 256, H, [300, 200], seed=13)  # dy [R, H]
    g = torch.Generator(device="cuda").manual_seed(17)
    w2 = (torch.randn(G, H, I, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    gu = torch.randn(R, 2 * I, generator=g, device="cuda").to(torch.bfloat16)
    dgu = torch.full((R, 2 * I), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_dgrad(dy, w2, off, dgu, swiglu_bwd_of=gu)
    gemm.check()
    for i in range(G):
        s, e = int(off[i]), int(off[i + 1])
        dact = (dy[s:e].float() @ w2[i].float()).to(torch.bfloat16).float()
        t = gu[s:e].float().view(e - s, I // 128, 2, 128)
        gt, ut = t[:, :, 0].reshape(e - s, I).requires_grad_(), t[:, :, 1].reshape(e - s, I).requires_grad_()
        (torch.nn.functional.silu(gt) * ut).backward(dact)
        got = dgu[s:e].float().view(e - s, I // 128, 2, 128)
        _close(got[:, :, 0].reshape(e - s, I), gt.grad)
        _close(got[:, :, 1].reshape(e - s, I), ut.grad)


@pytest.mark.parametrize("counts,N,K,granule,keep_counters", [
    ([1], 256, 64, 32, False),                                       # one tile of the narrowest width, one block
    ([1, 0, 2], 1024, 14336, 32, True),                              # few tiles: the reduction is cut as a stream, several parts per tile
    ([31, 32, 33, 255, 256, 257, 513], 512, 1024, 32, True),         # widths around the 32-row steps and the 256-token tile
    ([63, 64, 65, 1000, 2100], 768, 2048, 64, True),                 # several token tiles per group, of unequal width
    ([1030, 300], 1024, 8192, 64, True),                             # the same, forward reductions cut in equal parts
    ([1030, 300], 8192, 1024, 64, True),                             # ... and those of the data gradients
    ([(7 * i) % 70 for i in range(300)], 256, 256, 64, False),       # more groups than prefix entries
])
def test_live_rows_and_cut_reductions(counts, N, K, granule, keep_counters, kernel_variant):
    """Forward (plain, SwiGLU with and without the kept tiles) and dgrad (plain, SwiGLU backward) on the real rows only: those
    match fp32, the rows past their granule stay untouched. Twice with kept counters: they are clean for the next launch."""
    if kernel_variant != "cta_pair":
        pytest.skip("live rows belong to the CTA-pair kernels")
    from fast_b200.ops import gemm

    G = len(counts)
    counts_t, off, R, a, w = _setup(G, N, K, counts, seed=21)
    g = torch.Generator(device="cuda").manual_seed(23)
    live, scratch = counts_t.to(torch.int32), gemm.TokScratch(a.device) if keep_counters else None
    kw = dict(live_rows=live, granule=granule, scratch=scratch)
    new = lambda cols: torch.full((R, cols), 7.0, device="cuda", dtype=torch.bfloat16)
    dy = torch.randn(R, N, generator=g, device="cuda").to(torch.bfloat16)
    gu = torch.randn(R, 2 * K, generator=g, device="cuda").to(torch.bfloat16)
    for _ in range(2 if keep_counters else 1):
        out, act, act2, kept, dx, dgu = new(N), new(N // 2), new(N // 2), new(N), new(K), new(2 * K)
        gemm.grouped_gemm_fwd(a, w, off, out, **kw)
        gemm.grouped_gemm_fwd(a, w, off, act, swiglu=True, gate_up_out=kept, **kw)
        gemm.grouped_gemm_fwd(a, w, off, act2, swiglu=True, **kw)
        if K % 256 == 0:
            gemm.grouped_gemm_dgrad(dy, w, off, dx, **kw)
            gemm.grouped_gemm_dgrad(dy, w, off, dgu, swiglu_bwd_of=gu, **kw)
    gemm.check()
    o = off.tolist()
    for i in range(G):
        s, e, n = o[i], o[i + 1], counts[i]
        if n == 0:
            continue
        end = s + (n + granule - 1) // granule * granule
        full = a[s:s + n].float() @ w[i].float().T
        t = full.view(n, N // 256, 2, 128)
        _close(out[s:s + n], full)
        _close(kept[s:s + n], full)
        _close(act[s:s + n], (torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(n, N // 2))
        assert torch.equal(act[s:s + n], act2[s:s + n])
        assert all(bool((x[end:e] == 7).all()) for x in (out, act, act2, kept, dx, dgu))
        if K % 256 == 0:
            dact = dy[s:s + n].float() @ w[i].float()
            _close(dx[s:s + n], dact)
            q = gu[s:s + n].float().view(n, K // 128, 2, 128)
            gt, ut = q[:, :, 0].reshape(n, K).requires_grad_(), q[:, :, 1].reshape(n, K).requires_grad_()
            (torch.nn.functional.silu(gt) * ut).backward(dact.to(torch.bfloat16).float())
            got = dgu[s:s + n].float().view(n, K // 128, 2, 128)
            _close(got[:, :, 0].reshape(n, K), gt.grad)
            _close(got[:, :, 1].reshape(n, K), ut.grad)


@pytest.mark.parametrize("counts,N,K,granule,keep_counters", [
    ([1, 32, 255, 256, 257, 288, 289, 511, 512, 513, 545], 512, 1024, 32, True),   # one and two accumulators, every remainder at the edges
    ([300], 1024, 14336, 32, True),                                                 # cut as a stream: parts of both accumulators
    ([1030, 2100, 64], 768, 2048, 64, True),                                        # several wide tiles per group
    ([1030, 300], 1024, 8192, 64, True),                                            # the same, forward reductions cut in equal parts
    ([1030, 300], 8192, 1024, 64, True),                                            # ... and those of the data gradients
    ([(13 * i) % 600 for i in range(260)], 256, 256, 64, False),                    # more groups than prefix entries, tiles of one and of two
    ([700], 256, 64, 32, False),                                                    # a single block: nothing between the two ends of a tile
])
def test_wide_tiles(counts, N, K, granule, keep_counters, kernel_variant, monkeypatch):
    """The same on tiles of up to 512 tokens in two accumulators, whichever sizes the rule would take them for."""
    from fast_b200.ops import gemm

    monkeypatch.setattr(gemm, "wide_tiles", lambda *a: True)
    test_live_rows_and_cut_reductions(counts, N, K, granule, keep_counters, kernel_variant)


def test_the_sizes_above_take_the_paths_that_they_name():
    """What the work split makes of them on this GPU: streams, equal parts, and which passes they are in."""
    from fast_b200 import _C

    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    split = lambda rows, feats, red, tile_n, granule: _C.token_split(rows, feats // 256, red, tile_n, granule, pairs)
    for tile_n in (256, 512):
        for rows, N, K in (([1030, 300], 1024, 8192), ([1030, 300], 8192, 1024)):
            cut, whole = split(rows, min(N, K), max(N, K), tile_n, 64), split(rows, max(N, K), min(N, K), tile_n, 64)
            assert cut["shares"] > 1 and cut["cut_tiles"] > 0 and not cut["stream"] and whole["cut_tiles"] == 0
    for rows, tile_n in (([1, 0, 2], 256), ([300], 512)):
        stream = split(rows, 1024, 14336, tile_n, 32)
        assert stream["stream"] and stream["cut_tiles"] > 0 and stream["shares"] > stream["cut_tiles"]


@pytest.mark.parametrize("counts,N,K", [([0, 1, 64, 65, 128, 129, 192, 193], 256, 512), ([700, 0, 5000], 512, 1536), ([300, 200], 256, 768)])
def test_wgrad_of_few_and_many_blocks(counts, N, K, kernel_variant, monkeypatch):
    """Weight gradients in tiles of 512 columns (of 256 for 768 columns), with none, one, two ... blocks of 64 rows to reduce over."""
    from fast_b200.ops import gemm

    monkeypatch.setattr(gemm, "wide_columns", lambda row_tiles, columns, pairs, mean_rows: columns % 512 == 0)
    test_wgrad(len(counts), N, K, counts)


def test_wgrad_stops_at_the_live_rows(kernel_variant):
    """Rows past the next multiple of 64 are not read: what lies there (here NaN) does not reach the gradient."""
    from fast_b200.ops import gemm

    counts, N, K = [1, 64, 65, 0, 300], 256, 256
    counts_t, off, R, x, _ = _setup(5, 256, K, counts, seed=25)
    dy = torch.randn(R, N, generator=torch.Generator(device="cuda").manual_seed(27), device="cuda").to(torch.bfloat16)
    for i, n in enumerate(counts):
        s = int(off[i])
        x[s + (n + 63) // 64 * 64:int(off[i + 1])] = float("nan")
    out = torch.full((5, N, K), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_wgrad(dy, x, off, out, live_rows=counts_t.to(torch.int32))
    gemm.check()
    for i, n in enumerate(counts):
        s = int(off[i])
        _close(out[i], dy[s:s + n].float().T @ x[s:s + n].float())


@pytest.mark.parametrize("counts,N,K", [
    ([2049, 33], 4608, 8192),   # 2049 tokens in tiles of unequal width
    ([4097, 4096, 65], 2560, 2048),   # weight gradient: 65, 64 and 2 reduction blocks, 80 tiles each
])
def test_reductions_walked_backwards(counts, N, K, kernel_variant):
    """Sizes at which every other wave of the weight gradient walks the reduction from its end: forward and weight gradient equal the fp32 product."""
    if kernel_variant != "cta_pair":
        pytest.skip("belongs to the CTA-pair kernels")
    from fast_b200.ops import gemm

    G = len(counts)
    counts_t, off, R, a, w = _setup(G, N, K, counts, seed=29)
    live = counts_t.to(torch.int32)
    dy = torch.randn(R, N, generator=torch.Generator(device="cuda").manual_seed(31), device="cuda").to(torch.bfloat16)
    o = off.tolist()
    out, dw = torch.zeros(R, N, device="cuda", dtype=torch.bfloat16), torch.zeros_like(w)
    gemm.grouped_gemm_fwd(a, w, off, out, live_rows=live, granule=32)
    gemm.grouped_gemm_wgrad(dy, a, off, dw, live_rows=live)
    gemm.check()
    for i, n in enumerate(counts):
        s = o[i]
        _close(out[s:s + n], a[s:s + n].float() @ w[i].float().T)
        _close(dw[i], dy[s:s + n].float().T @ a[s:s + n].float())


@pytest.mark.parametrize("wide,counts,N,K,backwards", [(False, [1800, 33], 4608, 16384, [True, False]), (False, [1800, 33], 16384, 4608, [False, True]),
                                                      (True, [2100, 33], 9216, 8192, [True, True])])
def test_token_tiles_walked_backwards(wide, counts, N, K, backwards, kernel_variant, monkeypatch):
    """Sizes at which every other wave of the forward pass and of the data gradient walks the reduction from its end, with tiles of up to 256 and of
    up to 512 tokens: more token tiles than a band has, and whole tiles for more than one wave."""
    if kernel_variant != "cta_pair":
        pytest.skip("belongs to the CTA-pair kernels")
    from fast_b200 import _C
    from fast_b200.ops import gemm

    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    for (feats, red), back in zip(((N, K), (K, N)), backwards):
        s = _C.token_split(counts, feats // 256, red, 512 if wide else 256, 32, pairs)
        assert (s["token_tiles"] > s["back_tiles"] and s["token_tiles"] * (feats // 256) > s["cut_tiles"] + pairs) == back, s
    monkeypatch.setattr(gemm, "wide_tiles", lambda *a: wide)
    counts_t, off, R, a, w = _setup(len(counts), N, K, counts, seed=33)
    live = counts_t.to(torch.int32)
    dy = torch.randn(R, N, generator=torch.Generator(device="cuda").manual_seed(35), device="cuda").to(torch.bfloat16)
    out, dx = torch.zeros(R, N, device="cuda", dtype=torch.bfloat16), torch.zeros(R, K, device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_fwd(a, w, off, out, live_rows=live, granule=32)
    gemm.grouped_gemm_dgrad(dy, w, off, dx, live_rows=live, granule=32)
    gemm.check()
    for i, n in enumerate(counts):
        s = int(off[i])
        _close(out[s:s + n], a[s:s + n].float() @ w[i].float().T)
        _close(dx[s:s + n], dy[s:s + n].float() @ w[i].float())


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("counts,N,K", [([700, 0, 1030], 512, 512), ([1030, 300], 1024, 8192)])
def test_wide_tiles_wait_for_every_arrival_counter_that_they_touch(counts, N, K, swiglu, kernel_variant, monkeypatch):
    """A tile of up to 512 tokens takes two or three counters of 256 rows. With all rows in, the product is right; with one counter short of one row
    the launch gives up (whole tiles, and tiles whose reduction is cut), and the next one is as if it had not been."""
    if kernel_variant != "cta_pair":
        pytest.skip("belongs to the CTA-pair kernels")
    from fast_b200 import runtime
    from fast_b200.ops import gemm

    monkeypatch.setattr(gemm, "wide_tiles", lambda *a: True)
    counts_t, off, R, a, w = _setup(len(counts), N, K, counts, seed=37)
    live, o = counts_t.to(torch.int32), off.tolist()
    target = torch.zeros(R // 256, dtype=torch.int64)
    for i, n in enumerate(counts):
        for r in range(0, n, 256):
            target[(o[i] + r) // 256] = min(256, n - r)
    target = target.cuda()
    out = torch.zeros(R, N // 2 if swiglu else N, device="cuda", dtype=torch.bfloat16)
    want = []
    for i, n in enumerate(counts):
        full = a[o[i]:o[i] + n].float() @ w[i].float().T
        t = full.view(n, N // 256, 2, 128)
        want.append((torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(n, N // 2) if swiglu else full)
    for slot in [None, *range(R // 256), None]:
        counter = target.clone()
        if slot is not None:
            counter[slot] -= 1
        gemm.grouped_gemm_fwd(a, w, off, out.zero_(), swiglu=swiglu, live_rows=live, gate=(counter.data_ptr(), target), gate_tile_rows=256,
                              timeout_s=5.0 if slot is None else 0.02)
        if slot is None:
            gemm.check()
            for i, n in enumerate(counts):
                _close(out[o[i]:o[i] + n], want[i])
        else:
            with pytest.raises(runtime.CollectiveTimeout):
                gemm.check()
            gemm._st().clear()


def test_custom_operators_run_the_same_kernels():
    """torch.ops.fast_b200.* (schemas, mutation annotations) give the same bits as the direct calls."""
    from fast_b200.ops import gemm, registry  # noqa: F401

    G, N, K = 2, 512, 256
    counts, off, R, a, w = _setup(G, N, K, [200, 77], seed=5)
    direct = torch.zeros(R, N, device="cuda", dtype=torch.bfloat16)
    via_op = torch.zeros(R, N, device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_fwd(a, w, off, direct)
    torch.ops.fast_b200.grouped_gemm_fwd(a, w, off, via_op, False, None)
    gemm.check()
    assert torch.equal(direct, via_op)
    dx1, dx2 = torch.zeros_like(a), torch.zeros_like(a)
    gemm.grouped_gemm_dgrad(direct, w, off, dx1)
    torch.ops.fast_b200.grouped_gemm_dgrad(direct, w, off, dx2, None)
    dw1, dw2 = torch.zeros_like(w), torch.zeros_like(w)
    gemm.grouped_gemm_wgrad(direct, a, off, dw1)
    torch.ops.fast_b200.grouped_gemm_wgrad(direct, a, off, dw2)
    gemm.check()
    assert torch.equal(dx1, dx2) and torch.equal(dw1, dw2)
    logits = torch.randn(300, 16, device="cuda")
    idx, wts = torch.ops.fast_b200.route_topk(logits, None, 2)
    ref = torch.softmax(logits, -1).topk(2, dim=-1)
    assert torch.equal(idx.long(), ref.indices) and torch.allclose(wts, ref.values / ref.values.sum(-1, keepdim=True), atol=1e-5)


def _quant_e4m3_1x128(a):
    """bf16 [R, K] -> (uint8 e4m3 [R, K], fp32 scales [R, K/128]) with amax / 448 scales, and the dequantised fp32 matrix
    (rounded to bf16, which is what the kernel feeds the tensor core)."""
    R, K = a.shape
    g = a.float().view(R, K // 128, 128)
    sc = g.abs().amax(-1).clamp_min(1e-12) / 448.0
    sc = ((sc.view(torch.int32) + 0xFFFF) & ~0xFFFF).view(torch.float32)   # rounded up to bf16 precision, as the dispatch kernel does
    q = (g / sc.unsqueeze(-1)).to(torch.float8_e4m3fn)
    deq = (q.float() * sc.unsqueeze(-1)).to(torch.bfloat16).float().view(R, K)
    return q.view(R, K).view(torch.uint8).contiguous(), sc.contiguous(), deq


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("G,N,K,counts", [(1, 256, 128, [256]), (2, 512, 384, [200, 77]), (4, 768, 512, [0, 300, 128, 1])])
def test_forward_from_e4m3_rows(G, N, K, counts, swiglu, kernel_variant):
    """Operand A as e4m3 bytes + 1x128 scales, converted to bf16 tiles inside the kernel: equals the
    product of the dequantised matrix; rows past a group's real end count as zeros even when the
    buffer holds stale bytes and scales there."""
    if kernel_variant != "cta_pair":
        pytest.skip("the e4m3 operand feed belongs to the CTA-pair kernel")
    from fast_b200.ops import gemm

    counts_t, off, R, a, w = _setup(G, N, K, counts, seed=5)
    q, sc, deq = _quant_e4m3_1x128(a)
    # stale content in the pad rows: must not leak into anything
    real = torch.zeros(R, dtype=torch.bool, device="cuda")
    for i in range(G):
        real[int(off[i]):int(off[i]) + int(counts_t[i])] = True
    q[~real] = 0x7E                       # 448 in e4m3
    sc[~real] = 3.0e38
    out = torch.full((R, N // 2 if swiglu else N), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_fwd(q, w, off, out, swiglu=swiglu, a_scales=sc, group_rows=counts_t.to(torch.int32))
    gemm.check()
    for i in range(G):
        s, e = int(off[i]), int(off[i + 1])
        full = (deq[s:e] * real[s:e].unsqueeze(1)) @ w[i].float().T
        if swiglu:
            t = full.view(e - s, N // 256, 2, 128)
            full = (torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(e - s, N // 2)
        _close(out[s:e], full)
        assert float(out[s + int(counts_t[i]):e].float().abs().max() if e > s + int(counts_t[i]) else 0.0) == 0.0
