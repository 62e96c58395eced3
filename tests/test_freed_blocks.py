"""Blocks that katsu_cuda_free keeps for the next katsu_cuda_alloc: a block freed twice is refused, as the driver refuses
it, and must not be handed out twice."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 1 << 20])
def test_second_free_is_refused(ctx, count):
    from katsu_b200 import cabi

    block = ctx.alloc(count)
    ctx.free(block)
    with pytest.raises(cabi.KatsuCudaError):
        ctx.free(block)
    first, second = ctx.alloc(count), ctx.alloc(count)
    assert first != second
    ctx.free(first)
    ctx.free(second)
