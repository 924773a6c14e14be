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

import chemdata
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


def _two_premixed(spec, implicit, method):
    """two blocks of different sizes side by side, without an interface: a plane, factor or
    pivot taken from the other block would show"""
    mech = None if spec == 9 else chemdata.subset(chemdata.h2_air_9sp(), ["H2", "H", "O2", "O", "OH", "H2O", "N2"])
    a, b = (ostc.case_premixed_box(*n, mech=mech, seed=q) for n, q in (((18, 13, 9), 7), ((11, 16, 6), 8)))
    for f in b.faces:
        f.block = 1
    a.blocks, a.faces = a.blocks + b.blocks, a.faces + b.faces
    return ostc.make_steady(a, implicit_method=implicit, chem_src_method=method)


@pytest.mark.parametrize("implicit", [0, 1])
@pytest.mark.parametrize("method", [0, 1, 2])
@pytest.mark.parametrize("spec,generated", [(9, True), (9, False), (7, None)])
def test_batched_species_are_the_per_block_ones(spec, generated, method, implicit):
    """point-implicit chemistry (none, EPI, DA) through the tile tables: the mechanism's own
    kernels, the generic ones, and a species count that another kernel unit holds"""
    case = _two_premixed(spec, implicit, method)
    (r1, a), (r0, b) = _run(case, True, 3, generated), _run(case, False, 3, generated)
    assert np.isfinite(r0).all() and np.array_equal(r0, r1)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("implicit", [0, 1])
def test_batched_species_and_sst_are_the_per_block_ones(implicit):
    case = ostc.make_steady(ostc.case_mixing_layer(20, 17, 9, full_host=True, rans_model=2, wall=True),
                            implicit_method=implicit)
    (r1, a), (r0, b) = _run(case, True), _run(case, False)
    assert np.isfinite(r0).all() and np.array_equal(r0, r1)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
