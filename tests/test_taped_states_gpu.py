"""The states that the reverse pass recomputes with the taped step are the
forward pass's bit for bit on grids whose forward step runs another shape than
the tape: thin tiles, partial persistent tiles, 32 x 24 tiles and, in FP64, two
kernels.  With a checkpoint at every step no state is recomputed; the gradient
of longer segments must equal that one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,precision", [
    ((100, 100), 32), ((256, 256), 32), ((384, 256), 32), ((500, 300), 32), ((1000, 700), 32),
    ((701, 500), 32), ((1801, 1600), 32), ((100, 80), 64)])
def test_recomputed_states_equal_the_forward_pass(om_lib, size, precision):
    steps = 6
    rng = np.random.default_rng(9)
    dtype = np.float32 if precision == 32 else np.float64
    grads = []
    target = (1.5 + 0.1 * rng.standard_normal((size[1], size[0]))).astype(dtype)
    for every in (1, 3, steps):
        h = om_lib.Hydro(size, precision=precision, gamma=1.4)
        h.init_kh(7)
        h.set_scalar("cfl", 0.4)
        p = h.read("pressure")
        p[size[1] // 3, size[0] // 4] *= dtype(1.5)  # one cell sets the time step
        h.write("pressure", p)
        grads.append(h.adjoint_run(steps, target, checkpoint_every=every))
        h.close()
    for loss, grad in grads[1:]:
        assert loss == grads[0][0]
        for x, y in zip(grad, grads[0][1]):
            assert np.array_equal(x, y)
