"""The tiled reverse in both shapes: a context of one garment takes a tile with two groups of threads,
a batch with more tiles per color than the GPU has SMs with one.  Every copy in the batch has the
gradients of the garment alone, within the bounds of the batched adjoint's test.  Local colors of
a few elements and of more than a group has threads."""
import numpy as np
import pytest

pytest.importorskip("torch")

from xrtailor_gb300 import ClothSolver, scenes

pytestmark = pytest.mark.gpu

COPIES = 160  # more than the 152 SMs
KEYS = ("position", "velocity", "mass", "stretch_compliance", "bend_compliance")


@pytest.mark.parametrize("n", [6, 27])
def test_copies_have_the_gradients_of_one(xrt, n):
    p = scenes._params(num_substeps=2, num_iterations=2, stretch_compliance=1e-7,
                       bend_compliance=1e-3, enable_self_collision=0, num_collision_passes=2,
                       update_obstacle_animation=0)
    cloth = scenes.grid_cloth(n, 0.4, jitter=1e-3, seed=n)
    cloth.fixed_indices = scenes.two_corner_pins(n)
    rng = np.random.default_rng(n)
    v0 = rng.normal(0.0, 0.05, (n * n, 3)).astype(np.float32)
    c = rng.normal(size=(n * n, 3)).astype(np.float32)
    one, batch = ClothSolver(p), ClothSolver(p)
    one.add_cloth(cloth, particle_diameter=0.02)
    for _ in range(COPIES):
        batch.add_instance(cloth, None, particle_diameter=0.02)
    grads = []
    for s, k in ((one, 1), (batch, COPIES)):
        s.start()
        s.set_state(np.tile(cloth.positions, (k, 1)), np.tile(v0, (k, 1)))
        s.diff_begin()
        s.step()
        grads.append(s.backward(np.tile(c, (k, 1))))
    a, b = grads
    for key in KEYS:
        want = a[key]
        got = b[key].reshape((COPIES,) + want.shape)
        assert np.isfinite(want).all() and np.abs(want).max() > 0
        for k in (0, 77, COPIES - 1):
            np.testing.assert_allclose(got[k], want, rtol=2e-4, atol=2e-5 * np.abs(want).max(),
                                       err_msg=key)
