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


@pytest.mark.gpu
def test_depth_that_only_the_fp64_coarse_launch_holds(cmg):
    """64^3 in 4096 boxes of 4^3: the bottom depth fits the coarse launch in FP64 (217,088 of 225,280 bytes of shared
    memory) and not in FP32 (241,664, with the FP64 bottom vectors).  An FP32 cycle relaxes it without separate ghost
    fills all the same, and to the bits of the fills."""
    h = cmg.Hierarchy(64, boxes_of(cmg, 64, 4, 4), op=1, alpha=1.0, beta=-1.0)
    h.fill_synthetic(5, device=True)
    h.set_bottom_solver(imax=4)
    p = cmg.solve_params(iter_max=2)
    got = []
    for mode in (0, 1):
        h.set_relax_mode(mode)
        for mixed in (False, True):
            out = []
            fills = ghost_fills(h, lambda: out.append(h.solve(p, mixed=mixed)))
            assert (fills == 0) == (mode == 0), (mode, mixed, fills)
            got.append((out[0]["history"].tobytes(), h.phi(0).tobytes()))
    assert got[:2] == got[2:]
    h.close()


def grid_boxes(n0, size):
    return [[(x, y, z, x + size[0] - 1, y + size[1] - 1, z + size[2] - 1) for z in range(0, n0, size[2])
             for y in range(0, n0, size[1]) for x in range(0, n0, size[0])]]


@pytest.mark.gpu
@pytest.mark.parametrize("n0,size,op,bc,per,rest", [
    (180, (36, 12, 12), 0, "NDPPDN", 2, 1),  # 11 chunks of 256 cells of a colour per box, 12,375 in all
    (208, (16, 16, 16), 1, "DDDDDD", 3, 2),  # 8 per box, 17,576 in all
    (216, (24, 24, 24), 0, "PPPPPP", 4, 3),  # 27 per box, 19,683 in all
])
def test_blocks_of_several_chunks(cmg, n0, size, op, bc, per, rest):
    """Levels of more than 9472 chunks of a colour, where a block takes two to four of them (the last one fewer) and
    goes from one box to the next: sweeps, residual, its norm and the restriction against the filled ghosts."""
    nbox = (n0 // size[0]) * (n0 // size[1]) * (n0 // size[2])
    chunks = nbox * -(-size[0] // 2 * size[1] * size[2] // 256)
    assert min(4, chunks // (148 * 32)) == per and chunks % per == rest
    h = cmg.Hierarchy(n0, grid_boxes(n0, size), op=op, alpha=1.0, beta=-1.0 if op else -0.1, bc=bc)
    h.fill_synthetic(13, device=True)
    assert h.relax_variants()[0]["variant"] == "reads across faces"
    h.set_bottom_solver(imax=2)
    p = cmg.solve_params(pre=2, post=1, bottom=1, iter_max=2)
    for mixed in (False, True):
        got = []
        for mode in (0, 1):
            h.set_relax_mode(mode)
            out = h.solve(p, mixed=mixed)
            got.append((out["history"].tobytes(), h.phi(0).tobytes(), h.residual_norm()))
        assert got[0] == got[1], mixed
    h.close()
