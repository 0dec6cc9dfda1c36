"""What tells one cached launch plan of the expert GEMMs from another (no GPU)."""
import torch

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
