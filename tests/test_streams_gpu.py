"""Calls on a stream other than the current one."""
import inspect

import pytest

torch = pytest.importorskip("torch")

import llmt_b200 as L

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("call", [L.gemm, inspect.unwrap(L.gemm)], ids=["native", "python"])
def test_scratch_that_a_call_takes_belongs_to_its_stream(call):
    """Scratch of a call without a workspace is let go when the call is enqueued; memory of the current stream would be given
    to whoever allocates next, while the call on the other stream still uses it."""
    side = torch.cuda.Stream()
    a = torch.randn(2048, 256, device=DEV).bfloat16()
    b = torch.randn(2048, 256, device=DEV).bfloat16()
    c = torch.empty(256, 256, device=DEV)
    need = L.workspace_bytes(L.make_desc(c, a, b, True, False), a, b)
    assert need > 0
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    of_side = lambda: sum(s["total_size"] for s in torch.cuda.memory_snapshot() if s["stream"] == side.cuda_stream)
    assert of_side() == 0
    torch.cuda._sleep(1000000)
    side.wait_stream(torch.cuda.current_stream())
    call(c, a, b, True, False, stream=side)
    assert of_side() >= need
    over = torch.full((need // 4,), float("nan"), device=DEV)   # what the current stream gets next
    side.synchronize()
    want = a.double().T @ b.double()
    assert ((c.double() - want).norm() / want.norm()).item() < 1e-5
    del over
