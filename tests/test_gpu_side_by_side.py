"""Several contexts of one program mapping at the same time: blocks of one context's kernels share SMs with another's."""
import numpy as np
import pytest

from util import Context, make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    # neurons, id, nd, ed, R, mode: pairs of blocks two to an SM (three-stage rings), pairs whose few slices make small blocks that
    # fill the tensor memory two or three to an SM, uint16 and float32 pairs (a block fills it alone)
    (1000, 64, 60, 56, 360, 2), (300, 24, 16, 11, 360, 2), (300, 24, 16, 11, 360, 1), (300, 24, 16, 6, 360, 0),
])
def test_contexts_map_side_by_side(cuda, case):
    import pink_b200.capi as capi
    N, idim, nd, ed, R, mode = case
    n, rounds = 64, 30
    rng = np.random.default_rng(N + mode)
    contexts, inputs, outputs, want = [], [], [], []
    try:
        for k in range(3):
            ctx = Context(capi, make_config(capi, N, 1, idim, nd, ed, R, True, mode))
            contexts.append(ctx)
            ctx.set_som(rng.random((N, 1, nd, nd), dtype=np.float32))
            inputs.append(cuda.from_numpy(rng.random((n, 1, idim, idim), dtype=np.float32)).cuda())
            outputs.append((cuda.empty(n, N, device="cuda"), cuda.empty(n, N, dtype=cuda.int32, device="cuda")))
        cuda.cuda.synchronize()

        def start(k):
            contexts[k].e.map_device(inputs[k].data_ptr(), n, outputs[k][0].data_ptr(), outputs[k][1].data_ptr())

        for k in range(3):                                # one after the other
            start(k)
            contexts[k].e.synchronize()
            want.append([o.clone() for o in outputs[k]])
        for o in outputs:
            o[0].zero_(), o[1].zero_()
        cuda.cuda.synchronize()
        for _ in range(rounds):                           # and with nothing between them
            for k in range(3):
                start(k)
        for k in range(3):
            contexts[k].e.synchronize()
            assert cuda.equal(outputs[k][0], want[k][0]) and cuda.equal(outputs[k][1], want[k][1])
    finally:
        for ctx in contexts:
            ctx.close()
