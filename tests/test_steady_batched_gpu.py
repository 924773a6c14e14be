"""The steady iteration over several blocks: one tile-table launch per kernel
(DPLUR's first pass, sweeps and wall clearing, the update, the time step, the
residual partials) gives bitwise the blocks' own launches, for every number of
inner sweeps (the iterate's buffers swap roles with its parity, and without
sweeps dq is converted on its own), and the point-implicit chemistry of the
mechanism known at build time gives the generic tables' steady steps: an LU
with reciprocal pivots against one with quotients, within the 1e-9 that
either is held to against the oracle."""
import numpy as np
import pytest

import ostc

pytestmark = pytest.mark.gpu

LAYOUT = [((0, 0, 0), (20, 13, 10)), ((19, 0, 0), (37, 13, 10)), ((0, 12, 0), (20, 18, 10)), ((19, 12, 0), (37, 18, 10))]


def _run(case, batched, steps=2, generated=None):
    s, blocks = case.solver()
    s.set_batching(batched)
    if generated is not None:
        s.use_generated_chemistry(generated)
    s.initialize()
    res = s.steady_steps(steps, history=True)
    out = [b.download(n).copy() for b in blocks for n in ("bv", "dq")]
    s.close()
    return res, out


@pytest.mark.parametrize("sst", [0, 2])
@pytest.mark.parametrize("sweeps", [0, 1, 2, 3])
def test_batched_dplur_is_the_per_block_one(sst, sweeps):
    case = ostc.make_steady(ostc.case_uneven_blocks(layout=LAYOUT, rans_model=sst), implicit_method=1,
                            dplur_inner_step=sweeps)
    (r1, a), (r0, b) = _run(case, True), _run(case, False)
    assert np.isfinite(r0).all() and np.array_equal(r0, r1)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("implicit", [0, 1])
def test_generated_point_implicit_chemistry(implicit):
    case = ostc.make_steady(ostc.case_premixed_box(17, 12, 9), implicit_method=implicit)
    (r1, a), (r0, b) = _run(case, False, 4, True), _run(case, False, 4, False)
    assert np.max(np.abs(r1 - r0) / r0) <= 1e-9
    for x, y in zip(a, b):
        for l in range(x.shape[0]):
            assert np.max(np.abs(x[l] - y[l])) <= 1e-9 * np.max(np.abs(y[l]))
