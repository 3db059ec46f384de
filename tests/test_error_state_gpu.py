"""GPU: a refused call leaves nothing behind that fails the next one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_allocation_refused_by_the_runtime_does_not_fail_the_next_launch(ctx, kb, torch_cuda):
    torch = torch_cuda
    with pytest.raises(kb.KansoError):
        kb.KvPool(ctx, 64, 4_000_000, 16, 8, 128, kb.KV_INT8)  # 8.7 TB
    w = torch.from_numpy(np.zeros((8, 34), np.uint8)).cuda()
    x, y = torch.ones(1, 32, device="cuda"), torch.full((1, 8), 7.0, device="cuda")
    ctx.gemm_q8_0(w, x, y, 1, 8, 32, kb.ACT_F32)
    ctx.sync()
    assert (y == 0).all()
