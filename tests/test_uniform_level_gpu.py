"""Uniform levels (boxes side by side with boxes of the same shape), where the default relaxation rule reads neighbours
across box faces and the forced modes fill ghosts: the two give the same bits, also where a block takes several chunks
of cells, and a forced mode fills ghosts for the residual and the restriction as well as for the passes."""
import numpy as np
import pytest

GHOST = 2  # profile class of the ghost fills


def boxes_of(cmg, n0, max_box, block):
    return [cmg.domain_split((0, 0, 0), (n0 - 1,) * 3, max_box, block)]


def ghost_fills(h, call):
    h.profile_enable(True)
    call()
    n = h.profile_read(GHOST)[0]
    h.profile_enable(False)
    return n


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [False, True])
def test_forced_modes_fill_ghosts_for_residual_and_restriction(cmg, mixed):
    """64^3 in boxes of 32^3: five depths, the first four uniform.  Without sweeps a forced cycle fills for its four
    restrictions and the two residuals; the rule fills none of them."""
    h = cmg.Hierarchy(64, boxes_of(cmg, 64, 32, 8))
    h.fill_synthetic(3, device=True)
    h.set_bottom_grid(0)
    p = cmg.solve_params(pre=0, post=0, bottom=0, iter_max=1)
    for mode, solve, norm in ((0, 0, 0), (1, 6, 1), (2, 6, 1)):
        h.set_relax_mode(mode)
        assert ghost_fills(h, lambda: h.solve(p, mixed=mixed)) == solve, mode
        assert ghost_fills(h, h.residual_norm) == norm, mode
    h.close()
