"""Gradients of vertices that millions of paths add to.

The ground quad and the light of the displaced-sphere scene get up to 16.8M
contributions per term in 32-bit atomic adds. Which small ones are lost in the
large running sum depends on how many lanes' adds are summed first and in which
order paths end, so nearly cancelling components show a change of either far
above the difference of two runs (0.15 % of the gradient's RMS): sweeping paths
in the order in which they ended, and scattering boundary samples 32 at a time,
moved them by 0.9 %. The values are those of one thread per path in slot order
(mean of six runs).
"""
import pytest
import torch

from tensorray_b200 import api, scenes

pytestmark = pytest.mark.gpu

RMS = 13.380
HOT = [[8.924, -1798.614, 8.606], [6.064, -252.624, 9.384], [6.296, -2211.850, 1.316], [0.896, -639.758, -9.581],
       [1308.772, 269.399, 1077.543], [-1301.306, 269.949, 1073.951], [-1535.065, 40.740, -1757.394],
       [1518.704, 39.316, -1749.135]]


def test_sums_of_hot_vertices_keep_their_values(built_lib):
    sc = api.Scene(scenes.config2_scene(512, 512))
    sc.configure()
    sc.set_path_cache(16 << 30)
    o = api.RenderOptions(1, 5, 64, 64, 64, 64, 64)
    tracer = api.PathTracer()
    terms = [tracer, api.PrimaryEdgeIntegrator(), api.DirectEdgeIntegrator(), api.IndirectEdgeIntegrator(),
             api.PixelBoundaryIntegrator()]
    runs = 4
    total = torch.zeros(8, 3, dtype=torch.float64)
    for _ in range(runs):
        d = tracer.renderC(sc, o) - 0.3
        sc.clear_grads()
        for t in terms:
            t.renderD(sc, o, d)
        total += sc.get_grads()["positions"][-8:].double().cpu()
    ref = torch.tensor(HOT, dtype=torch.float64)
    scale = ref.abs().clamp_min(RMS)
    # the mean of four runs lies within 0.1 % of the values, the changes above at 0.9 %
    assert float(((total / runs - ref).abs() / scale).max()) < 3e-3
