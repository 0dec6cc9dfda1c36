"""What tells one cached launch plan of the expert GEMMs from another (no GPU)."""
import torch

from fast_b200.ops import gemm
from fast_b200.ops.gemm import _plan_key


def test_a_plan_belongs_to_one_geometry_type_and_device():
    w, x = torch.empty(2, 256, 256, dtype=torch.bfloat16), torch.empty(512, 256, dtype=torch.bfloat16)
    buf = torch.empty(512, 512, dtype=torch.bfloat16)
    out, gu = torch.empty(512, 128, dtype=torch.bfloat16), buf[:, :256]
    base = _plan_key(0, 1, 32, w, x, out, gu)
    assert base == _plan_key(0, 1, 32, w.view(2, 256, 256), x[:], out[:], buf[:, :256])   # another object, the same memory in the same way
    others = [
        _plan_key(0, 1, 32, w.transpose(1, 2), x, out, gu),                        # square weights, transposed view: same address and shape
        _plan_key(0, 1, 32, w.view(torch.float16), x, out, gu),
        _plan_key(0, 1, 32, w, x.view(torch.float16), out, gu),
        _plan_key(0, 1, 32, w, x.t().t()[:256], out, gu),
        _plan_key(0, 1, 32, w, x, out.view(torch.float16), gu),
        _plan_key(0, 1, 32, w, x, out[:256], gu),
        _plan_key(0, 1, 32, w, x, out, buf.view(-1)[: 512 * 256].view(512, 256)),  # the same address, another row pitch
        _plan_key(0, 1, 32, w, x, out, None),
        _plan_key(0, 1, 64, w, x, out, gu),
    ]
    assert all(k != base for k in others) and len(set(others)) == len(others)


def test_tiles_are_not_sized_by_a_capacity():
    """A step of fewer entries than experts counts as one row per expert, not as unknown; and where the number of rows is unknown and the matrix
    is a receive buffer, its capacity does not stand in for it."""
    from types import SimpleNamespace

    from fast_b200.parallel.ep import ExpertParallel

    engine = SimpleNamespace(scratch=SimpleNamespace(early=False), comm=SimpleNamespace(world=4), T=4096, K=2, El=32, granule=32)
    engine._mean_rows = lambda T: ExpertParallel._mean_rows(engine, T)
    for T in (0, 1, 3, 15, 16, 4096):
        rs = SimpleNamespace(topk_idx=torch.empty(T, 2), group_rows=torch.empty(32))
        live = ExpertParallel._live(engine, rs)
        assert live["mean_rows"] == max(1, T * 2 // 32)
        mean = gemm.group_rows_hint(live["mean_rows"], 32 * 1024, 32, live["live_rows"])
        tile = gemm.token_tile(gemm.STORE, 28672, live["most_rows"], mean, 32, 4096, 74)
        assert T == 4096 or tile == 256
    assert gemm.group_rows_hint(0, 8192, 8, None) == 1024 and gemm.group_rows_hint(0, 8192, 8, torch.empty(8)) == 0
    assert gemm.token_tile(gemm.STORE, 28672, 0, 0, 8, 4096, 74) == gemm.token_tile(gemm.SWIGLU, 4096, 0, 0, 8, 28672, 74) == 256


def test_wide_tiles_only_where_they_are_not_slower():
    """Sizes at which tiles of 512 tokens or columns were measured slower get tiles of 256, and those that they are for get them."""
    def tokens(epi, groups, features, reduction, rows):
        return gemm.token_tile(epi, reduction, 0, rows, groups, features, 74)

    assert tokens(gemm.SWIGLU, 2, 4096, 4096, 320) == tokens(gemm.SWIGLU, 16, 4096, 4096, 320) == 256      # 24 -> 48, 166 -> 174 us
    assert tokens(gemm.SWIGLU, 8, 28672, 4096, 440) == 256 and tokens(gemm.SWIGLU, 32, 4096, 7168, 320) == 512
    assert tokens(gemm.STORE, 8, 4096, 28672, 450) == tokens(gemm.STORE, 8, 4096, 28672, 560) == 256      # a training step of 1800 tokens 9944 -> 10307
    assert tokens(gemm.STORE, 8, 4096, 14336, 1024) == tokens(gemm.STORE, 2, 4096, 14336, 3000) == 256
    assert tokens(gemm.STORE, 8, 4096, 28672, 8192) == tokens(gemm.STORE, 8, 4096, 14336, 4096) == tokens(gemm.SWIGLU_BWD, 8, 14336, 4096, 8192) == 512
    columns = lambda groups, n, k, rows: gemm.wide_columns(groups * (n // 256), k, 74, rows)
    assert not any(columns(2, 1024, 1024, r) or columns(8, 1024, 1024, r) for r in (1, 16, 256, 400, 500, 600))   # 12 -> 16 us
    assert not any(columns(8, 4096, 14336, r) for r in (660, 1024, 1500)) and not columns(4, 2048, 2048, 600)
    assert all(columns(8, 4096, 14336, r) for r in (1, 256, 500, 600, 2048, 8192)) and columns(4, 2048, 2048, 256) and columns(8, 2048, 2048, 400)
    assert not columns(8, 2048, 768, 16)
