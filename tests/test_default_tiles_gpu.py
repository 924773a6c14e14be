"""The default tiles of a new solver (default_tiles, api.cu) choose between the
staged kernels and plane kernels of several register budgets by the scheme,
the species count and the size. Every choice evaluates the same face functions
in the same order, so the residual is bitwise that of one fixed plane tile
(4 rows, 1 chunk, 128 registers), at sizes on both sides of the rule's lines:
odd and even rows, one wave and many, segments that end short, species counts
that do and do not fit two staged CTAs per SM, grids whose CTAs are all resident
with every register, SST blocks of both parities."""
import numpy as np
import pytest

import chemdata
import ostc

pytestmark = pytest.mark.gpu

H2 = chemdata.h2_air_9sp


def _roe(case):
    case.scheme.inviscid_scheme = 2
    return case


CASES = {
    "air_one_wave": lambda: ostc.case_vortex(17, 15, 9, reconstruction=2, inviscid_scheme=3),
    "air_many": lambda: ostc.case_vortex(70, 41, 33, reconstruction=3, inviscid_scheme=4),
    "roe": lambda: ostc.case_vortex(65, 48, 25, reconstruction=2, inviscid_scheme=2),
    "aweno": lambda: ostc.case_vortex(64, 31, 16),
    "mix9_odd": lambda: ostc.case_mixing_layer(33, 41, 17),
    "mix9_even": lambda: ostc.case_mixing_layer(64, 30, 8),
    "mix9_planar": lambda: ostc.case_mixing_layer(97, 64, 1),
    "mix4": lambda: ostc.case_mixing_layer(31, 24, 15, mech=chemdata.h2_mixing_4sp()),
    "mix12": lambda: ostc.case_mixing_layer(40, 17, 16, mech=chemdata.with_inert_copies(H2(), "N2", 3)),
    "roe_mid": lambda: ostc.case_vortex(50, 40, 30, reconstruction=2, inviscid_scheme=2),
    "roe_one_wave": lambda: ostc.case_vortex(41, 33, 10, reconstruction=2, inviscid_scheme=2),
    "aweno_one_wave_2d": lambda: ostc.case_vortex(33, 500, 1),
    "mix9_roe_one_wave": lambda: _roe(ostc.case_mixing_layer(16, 17, 15)),
    "mix9_sst": lambda: ostc.case_mixing_layer(33, 24, 17, rans_model=2, wall=True),
    "sst_one_wave": lambda: ostc.case_uneven_blocks(layout=[((0, 0, 0), (31, 25, 21))], rans_model=2),
    "sst_odd_and_even": lambda: ostc.case_uneven_blocks(
        layout=ostc.block_layout(5, n_layers=1, n_cols=2, rows=(2, 2), extra_row=(0, 1), dims=(66, 50, 40),
                                 ranges=((16, 140), (12, 100), (10, 100)), anchors=False), rans_model=2),
    "sst_blocks": lambda: ostc.case_uneven_blocks(
        layout=ostc.block_layout(5, dims=(40, 30, 32), ranges=((8, 20), (8, 14), (8, 10)), anchors=False), rans_model=2),
}


@pytest.mark.parametrize("name", list(CASES))
def test_default_tiles_give_the_plane_kernels_residual(name):
    c = CASES[name]()
    out = []
    for fixed in (False, True):
        s, blocks = c.solver()
        if fixed:
            s.set_tiles([(4 | 2 << 8, 1)] * 3)
        s.initialize()
        s.compute_rhs()
        out.append([b.download("dq").copy() for b in blocks])
        s.close()
    assert all(np.isfinite(a).all() for a in out[0])
    assert all(np.array_equal(a, b) for a, b in zip(*out))
