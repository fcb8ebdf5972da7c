"""The admission estimate covers a context of many small affine elements, whose
constants (six numbers an element and level) weigh most against its points."""
import numpy as np
import pytest

import ssenss_b200 as S
from ssenss_b200.mesh import box_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape, n", [((24, 24, 24), 3), ((24, 24, 24), 5)])
def test_estimate_covers_affine_constants(shape, n):
    m = box_mesh(shape)
    ctx = S.Context(0)
    try:
        ctx.set_setup_options(no_dealias=True, no_particles=True)
        ctx.setup_mesh(m, n)
        ctx.set_precision("mixed")
        f = np.zeros((m.nel, n, n, n))
        f[0, 0, 0, 0], f[-1, -1, -1, -1] = 1.0, -1.0
        ctx.solve_poisson_cg(f, np.zeros_like(f), max_iter=1, history=False)
        assert ctx.memory_bytes() <= S.request_bytes(n, m.nel, "mixed")
    finally:
        ctx.close()
