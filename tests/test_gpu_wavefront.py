"""The wavefront's own edges: rounds, stream capture and growth of its buffers,
paths without a bounce, views that end inside a round."""
import pytest
import torch

from tensorray_b200 import api, scenes
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

TERMS = (api.TRN_PATH_TRACER, api.TRN_PRIMARY_EDGE, api.TRN_DIRECT_EDGE, api.TRN_INDIRECT_EDGE, api.TRN_PIXEL_EDGE)


def _scene(w=40, h=28):
    sc = api.Scene(scenes.config1_scene(w, h))
    sc.configure()
    return sc


def _views(sc, n=3, spp=(8, 21, 4)):
    cams = [api.Camera(c.pos, c.target, c.up, c.width, c.height, c.fov)
            for c in scenes.fibonacci_cameras(n, 4.0, [48], seed=2)]
    cams[1] = api.Camera(cams[1].pos, (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 60, 33, 45.0)
    return api.ViewSet(sc, cams, list(spp[:n]))


def test_image_does_not_depend_on_rounds_or_runs(built_lib):
    """Samples of a pixel are summed in slot order within a round, so an image
    repeats bit for bit; rounds only regroup the sum."""
    sc = _scene(128, 96)
    o = api.RenderOptions(5, 4, 40, 0, 0, 0, 0)
    a = api.PathTracer().renderC(sc, o).clone()
    assert torch.equal(a, api.PathTracer().renderC(sc, o))
    vs = _views(sc, 3, (64, 70, 50))
    opts = api.RenderOptions(5, 4, 0, 0, 0, 0, 0)
    ref = vs.render(api.TRN_PATH_TRACER, opts).clone()
    for cache in (0, 1 << 30):
        vs.set_path_cache(cache)
        img = vs.render(api.TRN_PATH_TRACER, opts, launch=api.launch_config(round_log2=16))
        # up to 70 additions of 32-bit values in another grouping
        torch.testing.assert_close(img, ref, rtol=70 * 2 ** -24, atol=1e-7)


@pytest.mark.parametrize("depth", [0, 1, 2, 9, 16])
def test_view_set_equals_single_views(built_lib, depth):
    """All terms of a view set, in rounds that end inside views, against one
    view at a time in one round."""
    sc = _scene()
    vs = _views(sc)
    opts = api.RenderOptions(3, depth, 0, 0, 0, 0, 0)
    d = torch.rand(vs.npix, 3, device=sc.device) - 0.3
    small = api.launch_config(round_log2=16)
    for term in TERMS:
        vs.render_grad(term, opts, d, launch=small)
        g = sc.get_grads()["positions"]
        for i, (c, s) in enumerate(zip(vs.cameras, vs.spps)):
            one = api.ViewSet(sc, [c], [s], seeds=[i])
            one.render_grad(term, opts, d[vs.offsets[i]:vs.offsets[i] + c.width * c.height])
        ref = sc.get_grads()["positions"]
        assert rel_l2(g, ref) <= 1e-5 if float(ref.abs().sum()) > 0 else float(g.abs().sum()) == 0


def test_capture_without_buffers_and_replay_after_growth(built_lib):
    """A forward render captured before any buffers exist runs one thread per
    path; one captured with buffers still replays after the set's buffers grew."""
    sc = _scene()
    opts = api.RenderOptions(3, 3, 0, 0, 0, 0, 0)
    vs, bare = _views(sc), _views(sc)
    out = torch.empty(vs.npix, 3, device=sc.device)
    ref = vs.render(api.TRN_PATH_TRACER, opts).clone()   # vs has its round buffers now
    bare.render(api.TRN_PRIMARY_EDGE, opts)              # uploads the view table, allocates none
    graphs = []
    for v in (bare, vs):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            v.render(api.TRN_PATH_TRACER, opts, out=out)
        graphs.append(g)
    for g in graphs:
        out.zero_()
        g.replay()
        torch.testing.assert_close(out, ref, rtol=1e-5, atol=1e-6)
    vs.reserve(8)  # the buffers that the second graph holds grow
    d = torch.rand(vs.npix, 3, device=sc.device) - 0.3
    for term in TERMS:
        vs.render_grad(term, opts, d)
    out.zero_()
    graphs[1].replay()
    torch.testing.assert_close(out, ref, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("depth", [1, 2, 3, 6, 16])
def test_late_bounces_give_the_same_in_either_form(built_lib, depth):
    """The bounces that the tail kernel runs begin earlier in a small round (here
    at the first) than in a large one (at the fifth of 3.1M samples): a small
    view's image is the same bit for bit alone and beside a large view, and its
    gradient but for the order of the adds."""
    sc = _scene()
    small = api.Camera((0.5, 1.5, 3.5), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 37, 23, 45.0)
    large = api.Camera((0.0, 0.0, 4.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 512, 512, 45.0)
    opts = api.RenderOptions(3, depth, 0, 0, 0, 0, 0)
    n = small.width * small.height
    gen = torch.Generator(device="cuda").manual_seed(depth)
    d1 = torch.rand(n, 3, generator=gen, device=sc.device) - 0.3
    for cache in (0, 1 << 32):
        got = []
        for cams, spps in (([small], [5]), ([small, large], [5, 12])):
            vs = api.ViewSet(sc, cams, spps, seeds=list(range(len(cams))))
            vs.set_path_cache(cache)
            img = vs.render(api.TRN_PATH_TRACER, opts)[:n].clone()
            d = torch.zeros(vs.npix, 3, device=sc.device)
            d[:n] = d1
            vs.render_grad(api.TRN_PATH_TRACER, opts, d)
            got.append((img, sc.get_grads()["positions"].clone()))
            sc.clear_grads()
        assert torch.equal(got[0][0], got[1][0])
        assert float(got[0][1].abs().sum()) > 0
        assert rel_l2(got[0][1], got[1][1]) <= 1e-5


@pytest.mark.parametrize("w,h,spp,round_log2", [(8, 8, 31, 0), (8, 8, 32, 0), (8, 8, 33, 0), (1, 1, 4099, 0), (5, 3, 7001, 16),
                                                (128, 128, 33, 0), (129, 128, 33, 0), (8, 6, 3000, 16)])
def test_pixels_of_many_samples(built_lib, w, h, spp, round_log2):
    """A warp sums a pixel of 32 samples and more in a view of up to 16,384
    pixels: against one thread per path, which a capture without round buffers
    runs, in whole rounds and in some that end inside a pixel's samples, with a
    view of the other kind beside it, and the same bit for bit in two runs."""
    sc = _scene()
    cams = [api.Camera((0.5, 1.5, 3.5), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 40, 28, 45.0),
            api.Camera((0.0, 0.5, 4.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), w, h, 45.0)]
    opts = api.RenderOptions(3, 3, 0, 0, 0, 0, 0)
    bare, vs = api.ViewSet(sc, cams, [7, spp]), api.ViewSet(sc, cams, [7, spp])
    bare.render(api.TRN_PRIMARY_EDGE, opts)              # uploads the view table, allocates none
    ref = torch.empty(bare.npix, 3, device=sc.device)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        bare.render(api.TRN_PATH_TRACER, opts, out=ref)
    ref.zero_()
    g.replay()
    launch = api.launch_config(round_log2=round_log2) if round_log2 else None
    img = vs.render(api.TRN_PATH_TRACER, opts, launch=launch).clone()
    # spp additions of 32-bit values in another order
    torch.testing.assert_close(img, ref, rtol=spp * 2 ** -24 + 1e-6, atol=1e-7)
    assert torch.equal(img, vs.render(api.TRN_PATH_TRACER, opts, launch=launch))


def test_direct_set_up_in_either_form(built_lib):
    """Rounds of up to 2^19 slots run the direct set-up in one kernel, larger ones
    as a wavefront: one round of 2^19 + 4,096 slots against the same in rounds of
    2^16, and one of 2^19."""
    sc = _scene(64, 64)
    opts = api.RenderOptions(3, 3, 0, 0, 0, 0, 0)
    for spp in (128, 129):
        vs = api.ViewSet(sc, [api.Camera((0.5, 1.5, 3.5), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 64, 64, 45.0)], [spp])
        d = torch.rand(vs.npix, 3, device=sc.device) - 0.3
        got = []
        for launch in (None, api.launch_config(round_log2=16)):
            vs.render_grad(api.TRN_DIRECT_EDGE, opts, d, launch=launch)
            got.append(sc.get_grads()["positions"].clone())
        assert float(got[0].abs().sum()) > 0
        assert rel_l2(got[0], got[1]) <= 1e-5


@pytest.mark.parametrize("term,guided", [(t, False) for t in TERMS] + [(api.TRN_DIRECT_EDGE, True)])
def test_captured_gradients_replay_after_growth(built_lib, term, guided):
    """A captured gradient call holds the set's round and sort buffers, and a
    guided one the scene's tree: it still replays after a larger call grew them."""
    sc = _scene()

    def options(size):
        o = api.RenderOptions(3, 3, 0, 0, 0, 0, 0)
        o.g_direct, o.g_direct_depth, o.g_direct_max_size, o.g_direct_spp = guided, 1, size, 4
        return o

    vs = _views(sc)
    d = torch.rand(vs.npix, 3, device=sc.device) - 0.3
    sc.clear_grads()
    vs.render_grad(term, options(3000), d)               # allocates what this call needs
    ref = sc.get_grads()["positions"].clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        vs.render_grad(term, options(3000), d)
        got = sc.get_grads()["positions"]
    vs.reserve(8)
    large = _views(sc, 3, (90, 90, 90))
    for s in (vs, large):
        for t in TERMS:
            s.render_grad(t, options(90_000), d)
    junk = [torch.full((1 << 22,), float("nan"), device=sc.device) for _ in range(64)]  # over memory given back
    sc.clear_grads()
    g.replay()
    del junk
    assert float(ref.abs().sum()) > 0
    assert rel_l2(got, ref) <= 1e-5
