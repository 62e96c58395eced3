"""Adjoints that pass through unchanged (Add, Reshape) share one device buffer; a later contribution or a second backward
must not reach the other holders (crates/katsu-core/src/tensor.rs:353-356, 383-409).  Against the oracle graph, whose
adjoints are all separate; sums and products of small integers, so every value is exact and compared bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph(lib, backwards):
    values = {name: np.arange(i, i + 12, dtype=np.float32) % 5 - 2 for i, name in enumerate("abc")}
    t = {name: lib.Tensor(v, [3, 4]) for name, v in values.items()}
    if hasattr(t["a"], "reshape"):
        t["r"] = t["a"].reshape([3, 4])
    else:
        t["r"] = t["a"]
    t["s"] = t["r"].add(t["b"])        # r, b share s's adjoint
    t["p"] = t["s"].mul(t["c"])
    t["u"] = t["s"].add(t["p"])        # s receives u's adjoint, then p's contribution
    t["v"] = t["u"].add(t["b"])        # b: shared, then added to
    t["w"] = t["v"].add(t["v"])        # both edges to one parent
    t["loss"] = t["w"].sum()
    for _ in range(backwards):
        t["loss"].backward()
    return t


@pytest.mark.parametrize("backwards", [1, 3])
def test_gradients_are_independent(oracle, backwards):
    import katsu_b200 as K

    dev, ref = graph(K, backwards), graph(oracle, backwards)
    for name in ref:
        want = ref["a"].grad() if name == "r" and ref["r"] is ref["a"] else ref[name].grad()
        assert np.array_equal(np.asarray(dev[name].grad()).reshape(-1), np.asarray(want).reshape(-1)), name
    dev["v"].zero_grad()
    assert dev["v"].grad() is None and dev["u"].grad() is not None


def test_a_gradient_changed_in_place_is_one_tensors_own():
    """A caller that scales or reduces gradients through their device addresses must not reach another tensor's, nor the seed of
    later backward passes."""
    import katsu_b200 as K
    from katsu_b200 import cabi

    def overwrite(tensor, value):
        address = tensor.device_grad()
        K.synchronize()
        with cabi.Context(0) as context:
            context.h2d(address, np.full(tensor.numel(), value, np.float32))
            context.sync()

    values = np.arange(12, dtype=np.float32)
    a, b = K.Tensor(values, [3, 4]), K.Tensor(values + 1, [3, 4])
    total = a.add(b)
    loss = total.sum()
    loss.backward()
    overwrite(a, 7.0), overwrite(loss, 5.0)
    assert (np.asarray(a.grad()) == 7).all() and (np.asarray(loss.grad()) == 5).all()
    assert (np.asarray(b.grad()) == 1).all() and (np.asarray(total.grad()) == 1).all()
    for t in (a, b, total, loss):
        t.zero_grad()
    loss.backward()
    assert (np.asarray(a.grad()) == 1).all() and (np.asarray(loss.grad()) == 1).all()
