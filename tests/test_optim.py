"""Host side of the fused optimizer (no GPU): what goes into one launch."""
import torch

from fast_b200 import runtime
from fast_b200.utils import FusedAdamW


def test_a_parameter_listed_twice_is_updated_one_launch_after_the_other(monkeypatch):
    """Tensors of one launch are updated side by side; the two updates of a tied parameter must not be."""
    launches = []

    class _Ext:
        @staticmethod
        def adamw_step(params, masters, ms, vs, grads, steps, *rest):
            launches.append([(p.data_ptr(), step) for p, step in zip(params, steps)])

    monkeypatch.setattr(runtime, "ext", lambda: _Ext)
    p, q = (torch.nn.Parameter(torch.zeros(16, dtype=torch.bfloat16)) for _ in range(2))
    p.grad, q.grad = torch.ones_like(p), torch.ones_like(q)
    FusedAdamW([p, q]).step()
    assert launches == [[(p.data_ptr(), 1), (q.data_ptr(), 1)]]
    launches.clear()
    FusedAdamW([p, q, p]).step()
    assert [x for batch in launches for x in batch if x[0] == p.data_ptr()] == [(p.data_ptr(), 1), (p.data_ptr(), 2)]
    assert all(len({a for a, _ in batch}) == len(batch) for batch in launches)
