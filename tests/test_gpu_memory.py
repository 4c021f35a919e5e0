"""Device memory: the scratch of float32 training's estimate holds what the split of one image needs, and less where the
device has no more; a context outlives a call that the memory did not suffice for."""
import numpy as np
import pytest

import oracle as O
from pink_b200.synthetic import blob_images
from util import Context, make_config

pytestmark = pytest.mark.gpu

SIDE0, SIDE1, IDIM, ND, ED, R = 20, 50, 40, 28, 20, 720
N, T, K = SIDE0 * SIDE1, 2 * R, ED * ED
KP = (K + 31) // 32 * 32
PLANE = N * T * 4                     # bytes of one image's dot products: 5.8 MB
MB = 1 << 20


def _context(capi, options=None):
    ctx = Context(capi, make_config(capi, N, 1, IDIM, ND, ED, R, True, 0), options)
    rng = np.random.default_rng(3)
    ctx.set_som(rng.random((N, 1, ND, ND), dtype=np.float32))
    ctx.set_factors(O.update_factors(0, SIDE0, SIDE1, O.FUNC_GAUSSIAN, 1.1, 0.2))
    return ctx


def _images(torch):
    return torch.from_numpy(np.ascontiguousarray(blob_images(4, IDIM, 1, seed=1), dtype=np.float32)).cuda()


def _train(ctx, images):
    ctx.e.train_device(images.data_ptr(), 4)
    return list(ctx.e.bmu_log(4)), ctx.get_som(np.zeros((N, 1, ND, ND), np.float32))


def _taken(torch, capi, options=None):
    """Bytes the first training call of a context takes."""
    images = _images(torch)
    with _context(capi, options) as ctx:
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        result = _train(ctx, images)
        return before - torch.cuda.mem_get_info()[0], result


def test_training_scratch_is_what_the_split_needs(cuda):
    import pink_b200.capi as capi
    for options in ({"f32_filter": 0}, None):
        _taken(cuda, capi, options)                       # kernels loaded
    without, _ = _taken(cuda, capi, {"f32_filter": 0})
    with_estimate, _ = _taken(cuda, capi)
    operands = 2 * 4 * KP * (N + T)                       # word planes of map and transforms
    # 35 tiles of 128 x 256: a handful of ranges fills the GPU (and the allocator gives whole 2 MB)
    assert with_estimate - without <= operands + 4 * PLANE + 16 * MB


def test_training_makes_do_with_less_scratch(cuda):
    """A split into fewer ranges where the memory for all of them is not there; the trained map is the same."""
    import pink_b200.capi as capi
    _taken(cuda, capi)
    taken, (bmus, som) = _taken(cuda, capi)
    images = _images(cuda)
    with _context(capi) as ctx:
        cuda.cuda.empty_cache()
        free = cuda.cuda.mem_get_info()[0]
        hog = cuda.empty(free - (taken - 3 * MB // 2), dtype=cuda.uint8, device="cuda")     # the split of this geometry has two planes
        try:
            got_bmus, got_som = _train(ctx, images)
        finally:
            del hog
            cuda.cuda.empty_cache()
    assert got_bmus == bmus
    assert np.array_equal(got_som.view(np.uint32), som.view(np.uint32))


@pytest.mark.parametrize("mode", [0, 2])
def test_context_outlives_a_refused_call(cuda, mode):
    """Mapping needs larger buffers than training; where they cannot be had the call is refused, and the next calls -- training
    first, whose smaller buffers went with the attempt -- find everything they need."""
    import pink_b200.capi as capi
    imgs = blob_images(4, IDIM, 1, seed=2).reshape(4, 1, IDIM, IDIM)
    d_imgs = cuda.from_numpy(np.ascontiguousarray(imgs, dtype=np.float32)).cuda()
    rng = np.random.default_rng(5)
    som0 = rng.random((N, 1, ND, ND), dtype=np.float32)
    F = O.update_factors(0, SIDE0, SIDE1, O.FUNC_GAUSSIAN, 1.1, 0.2)

    def run(starve):
        with Context(capi, make_config(capi, N, 1, IDIM, ND, ED, R, True, mode)) as ctx:
            ctx.set_som(som0)
            ctx.set_factors(F)
            ctx.e.train_device(d_imgs.data_ptr(), 4)
            ctx.e.synchronize()
            if starve:
                cuda.cuda.empty_cache()
                free = cuda.cuda.mem_get_info()[0]
                hog = cuda.empty(free - 24 * MB, dtype=cuda.uint8, device="cuda")
                try:
                    with pytest.raises(Exception, match="memory"):
                        ctx.map(imgs)
                finally:
                    del hog
                    cuda.cuda.empty_cache()
            ctx.e.train_device(d_imgs.data_ptr(), 4)
            bmus = list(ctx.e.bmu_log(4))
            som = ctx.get_som(som0)
            return bmus, som, ctx.map(imgs)

    want, got = run(False), run(True)
    assert want[0] == got[0]
    for a, b in ((want[1], got[1]), (want[2][0], got[2][0]), (want[2][1], got[2][1])):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
