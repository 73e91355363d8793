"""Scenes at the edges of what the marches assume: opacities of every sign, maps whose
cells rounding makes empty, and the launch choices such scenes decide.

Bars: maps and sample counts equal the oracle's, every launch choice gives the same
image bit for bit (not-a-number included), and images stay within the exact form's bar
(max |dRGBA| <= 2e-3, >= 99.9% of pixels identical).
"""
import dataclasses

import numpy as np
import pytest

from oracle.oracle import Oracle
from pilot_b200 import scenes
from test_marches_gpu import LIGHTS, frame, renderer, same, sparse
from test_rectilinear_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nextra", [0, 2])
def test_opacities_that_are_never_positive(cuda_device, nextra):
    """No positive opacity: the maps are 0, but the view march composites the negative ones."""
    dims = (33, 20, 25)
    s = dataclasses.replace(scenes.small(41, n=24, image=48, m=9, kind="noise"), dims=dims, array=sparse(dims, 9))
    s.tf = s.tf.copy()
    s.tf[:, 3] = np.where(np.arange(len(s.tf)) < 90, 0.0, -0.1)
    with renderer(s) as r:
        for kind, v in LIGHTS[:nextra]:
            (r.add_directional_light if kind else r.add_point_light)(v, (0.3, 0.9, 0.5), 0.7)
        r.set_multi_light(nextra > 0)
        out = []
        for skip in (False, True):
            r.set_tuning(empty_skip=skip, view_skip=skip)
            img, t = r.render(s.camera())
            out.append((img, r.get_shadow_map((nextra + 1) * 1000), (t["light_samples"], t["lit_samples"])))
        assert np.min(out[0][0][..., 3]) < 0
        same(out[1], out[0], "leaps")
    if nextra == 0:
        oimg, lit = Oracle(s).view_march(Oracle(s).light_march()[0])
        assert out[1][2][1] == lit
        check(out[1][0], oimg)
