"""Ray counts around a warp's 32 and scenes with and without a hierarchy of their own.

Point and directional lights and one ray a pixel: every pixel is the same function on both
sides, so a pixel may only differ where a ray grazes an edge (one pixel, or 0.5% of them,
further off than 1e-3 of its value).
"""
from __future__ import annotations

import numpy as np
import pytest

from fluid_gb300 import render as R
from tests.test_gpu_render import _case, _gpu, _tessellate, pbf  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("surface", [True, False])
@pytest.mark.parametrize("width,height,split", [(1, 1, 1), (31, 1, 1), (32, 1, 1), (33, 1, 2), (127, 5, 1), (65, 9, 2)])
def test_ragged_ray_counts(pbf, oracle_lib, width, height, split, surface):  # noqa: F811
    from oracle import oracle

    g, scene, cam, prm = _case("render_p_default")
    if split > 1:
        scene = _tessellate(scene, split)
        assert len(scene.tri) > 32
    scene.lights = [R.Light(R.POINT, (1.5, 1.2, 1.0), position=(-0.3, 1.2, 0.4)),
                    R.Light(R.DIRECTIONAL, (0.4, 0.4, 0.5), direction=(0.2, -1.0, -0.3))]
    out, sx, sn = _gpu(pbf, g, scene, cam, prm, width, height, 1, 0, 1, 5, surface)
    ref = oracle.render(scene, cam, sx, sn, width, height, 1, 0, 1, oracle.RNG_COUNTER, 5)
    d = np.abs(out["hdr"] - ref["hdr"]).max(-1)
    far = d > 1e-3 * np.maximum(np.abs(ref["hdr"]).max(-1), 1e-2) + 1e-4
    assert far.sum() <= max(1, 0.005 * far.size)
