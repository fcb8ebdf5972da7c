"""ssg_tuning after the autotuner has timed a context whose derivative matrices
lack the points' antisymmetry: the plane form in use, not the line form those
levels cannot take.  (Launch shapes are process-wide, so this runs late.)"""
import numpy as np
import pytest

import ssenss_b200 as S
from ssenss_b200.mesh import box_mesh

pytestmark = pytest.mark.gpu


def test_tuned_plane_form_is_reported():
    m = box_mesh((3, 3, 3))
    rng = np.random.default_rng(1)
    ctx = S.Context(0)
    ctx.setup_connectivity(m.neigh)
    orders = [7, 4, 2]
    for level, n in enumerate(orders):
        interp = None if level == 0 else rng.standard_normal((n, orders[level - 1]))
        ctx.setup_level(level, n, rng.standard_normal((n, n)), None, rng.uniform(0.1, 1.0, n),
                        rng.uniform(0.5, 1.5, (6, m.nel, n, n, n)),
                        rng.uniform(0.5, 1.5, (m.nel, n, n, n)), interp)
    ctx.setup_finish()
    shapes = ctx.autotune(reps=2)
    for n in (7, 4):
        assert shapes[n]["ax_elements_per_block"] >= 1
    ctx.close()
