"""The coarse cluster launch (depths and bottom solve in shared memory) and the passes that read across box faces on
uniform levels, against the launched path (ghost fills before every pass, relaxation mode 1; the bottom solve in one
block): same residual history and phi, bit for bit, at the sizes where their tables and splits change -- one box, boxes
that stop coarsening early, more than 512 boxes, depths on both sides of the one-block limit, walls, outflow and
periodic faces, V- and W-cycles, FP64 and mixed, both bottom solvers."""
import numpy as np
import pytest


def boxes_of(cmg, n0, max_box, block):
    return [cmg.domain_split((0, 0, 0), (n0 - 1,) * 3, max_box, block)]


def both(cmg, h, params, mixed, phi):
    out = []
    for mode, bottom in ((0, -1), (1, 0)):
        h.set_relax_mode(mode)
        h.set_bottom_grid(bottom)
        r = h.solve(params, mixed=mixed)
        out.append((r["exit_status"], r["history"].tobytes(), [p.tobytes() for p in phi()]))
    return out


CASES = [  # n0, max_box, block, op, bc
    (8, 8, 4, 0, "DDDDDD"), (16, 16, 8, 1, "DDDDDD"), (24, 24, 8, 0, "NNNNND"), (24, 12, 4, 1, "NDNDND"),
    (32, 16, 8, 1, "DDDDDD"), (32, 32, 8, 0, "PPNNDD"), (36, 12, 4, 0, "PPPPPP"), (40, 32, 8, 1, "DDDDDD"),
    (40, 4, 4, 0, "DDDDDD"), (48, 24, 8, 0, "PPPPPP"), (52, 20, 4, 0, "NNNNND"), (64, 32, 8, 1, "PPDDNN"),
]


@pytest.mark.gpu
@pytest.mark.parametrize("n0,max_box,block,op,bc", CASES)
def test_coarse_launch_matches_the_launched_path(cmg, n0, max_box, block, op, bc):
    alpha, beta = (1.0, -1.0) if op else ((1.0, -0.1) if bc == "PPPPPP" else (0.0, 1.0))
    h = cmg.Hierarchy(n0, boxes_of(cmg, n0, max_box, block), op=op, alpha=alpha, beta=beta, bc=bc)
    h.fill_synthetic(7, device=True)
    for kind in (0, 1):
        h.set_bottom_solver(kind=kind)
        for mixed in (False, True):
            for num_mg in (1, 2):
                p = cmg.solve_params(num_mg=num_mg, iter_max=3)
                a, b = both(cmg, h, p, mixed, lambda: [h.phi(0)])
                assert a == b, (kind, mixed, num_mg)
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n0,max_box,block,op,bc", [(60, 20, 4, 0, "DDDDDD"), (64, 20, 4, 1, "NDNDND"),
                                                    (64, 20, 4, 0, "PPPPPP")])
def test_large_bottoms_in_the_coarse_launch(cmg, n0, max_box, block, op, bc):
    """Bottom levels of 30^3 and 32^3 cells: more cells of a colour than the threads of a block hold in registers
    (1024; 1000 and 1100 on the fullest of 16 blocks)."""
    h = cmg.Hierarchy(n0, boxes_of(cmg, n0, max_box, block), op=op, alpha=1.0, beta=-1.0 if op else -0.1, bc=bc)
    h.fill_synthetic(9, device=True)
    assert [v["variant"] for v in h.relax_variants()][-1] == "coarse launch"
    for kind in (0, 1):
        h.set_bottom_solver(kind=kind, imax=5)
        for mixed in (False, True):
            a, b = both(cmg, h, cmg.solve_params(iter_max=2), mixed, lambda: [h.phi(0)])
            assert a == b, (kind, mixed)
            h.set_relax_mode(0)
            h.set_bottom_grid(-1)
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n0,max_box,op,first", [(32, 16, 0, 1), (48, 24, 0, 1), (32, 16, 1, 1), (48, 24, 1, 2)])
def test_first_depth_of_the_coarse_launch(cmg, n0, max_box, op, first):
    """Depths above the bottom join up to 25,000 cells (12,000 with variable coefficients): a 32^3 one never, a 24^3
    one with constant coefficients."""
    h = cmg.Hierarchy(n0, boxes_of(cmg, n0, max_box, 8), op=op, alpha=1.0, beta=-1.0 if op else -0.1)
    got = [v["variant"] == "coarse launch" for v in h.relax_variants()]
    assert got == [d >= first for d in range(len(got))]
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n0,max_box,op", [(16, 16, 1), (24, 16, 0), (40, 32, 1)])
def test_coarse_launch_in_refined_hierarchies_and_forests(cmg, n0, max_box, op):
    grids = [cmg.synthetic_hierarchy(n0, 2, max_box=max_box, seed=s) for s in (3, 4, 5)]
    h = cmg.Hierarchy(n0, grids[0], op=op, alpha=float(op), beta=-1.0 if op else 1.0)
    h.fill_synthetic(11, device=True)
    for mixed in (False, True):
        for num_mg in (1, 2):
            p = cmg.solve_params(num_mg=num_mg, iter_max=3)
            a, b = both(cmg, h, p, mixed, lambda: [h.phi(l) for l in range(h.nlev)])
            assert a == b, (mixed, num_mg)
    h.close()
    f = cmg.Forest(n0, grids, op=op, alpha=float(op), beta=-1.0 if op else 1.0)
    f.fill_synthetic([21, 22, 23])
    for mixed in (False, True):
        got = []
        for mode, bottom in ((0, -1), (1, 0)):
            f.set_relax_mode(mode)
            f.set_bottom_grid(bottom)
            r = f.solve(cmg.solve_params(iter_max=3), mixed=mixed)
            got.append(([x["final_norm"] for x in r], [f.phi(k, l).tobytes() for k in range(3) for l in range(2)]))
        assert got[0] == got[1], mixed
    f.close()


@pytest.mark.gpu
def test_nan_right_hand_side_ends_the_solve(cmg):
    """The residual's norm keeps a NaN, whether folded into the residual's pass or not: the solve ends before its first
    cycle, diverged."""
    h = cmg.Hierarchy(32, boxes_of(cmg, 32, 16, 8))
    rhs = np.ones(32 ** 3)
    rhs[1234] = np.nan
    h.set_rhs(0, rhs)
    for mode, bottom in ((0, -1), (1, 0)):
        h.set_relax_mode(mode)
        h.set_bottom_grid(bottom)
        r = h.solve(cmg.solve_params())
        assert r["diverged"] and r["iterations"] == 0
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind,norm_type", [(0, 0), (0, 2), (1, 0), (1, 2)])
@pytest.mark.parametrize("n0,max_box,block", [(32, 16, 8), (52, 20, 4)])
def test_overflow_in_the_bottom_solve(cmg, n0, max_box, block, kind, norm_type):
    """Right-hand sides from 1e153 to 1e160: the sums of squares in the bottom solve overflow.  With the max norm (and a
    breakdown threshold below zero) BiCGStab's scalars become NaN, and so do its vectors and norms; with the 2-norm the
    norms are infinite; in FP32 the cycle starts from infinities.  One block (2^3 cells a box) and all ranks (26^3
    cells) end as the launched bottom solve does, diverged if phi holds a NaN."""
    h = cmg.Hierarchy(n0, boxes_of(cmg, n0, max_box, block))
    rhs = 1.0 + 0.01 * np.random.default_rng(n0).standard_normal(n0 ** 3)
    h.set_bottom_solver(kind=kind, norm_type=norm_type, small=-1.0)
    for mixed in (False, True):
        nan = 0
        for scale in (1e153, 1e156, 1e160):
            h.set_rhs(0, scale * rhs)
            got = []
            for mode, bottom in ((0, -1), (1, 0)):
                h.set_relax_mode(mode)
                h.set_bottom_grid(bottom)
                r = h.solve(cmg.solve_params(iter_max=1), mixed=mixed)
                got.append((r["exit_status"], r["diverged"], np.asarray(r["history"]), h.phi(0)))
            assert got[0][:2] == got[1][:2], (mixed, scale)
            assert np.array_equal(got[0][2], got[1][2], equal_nan=True)
            assert np.array_equal(got[0][3], got[1][3], equal_nan=True)
            assert got[0][1] == np.isnan(got[0][3]).any()
            nan += got[0][1]
        assert nan or not (mixed or (kind, norm_type) == (0, 0))
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n0,levels,op", [(32, 1, 0), (32, 1, 1), (24, 2, 1)])
def test_coefficients_changed_between_solves(cmg, n0, levels, op):
    """The coarse launch's scalars and coefficients follow alpha and beta (graphs captured with other ones included) and
    new coefficient fields, in FP64 and mixed."""
    boxes = cmg.synthetic_hierarchy(n0, levels, max_box=16, seed=4) if levels > 1 else boxes_of(cmg, n0, 16, 8)
    h = cmg.Hierarchy(n0, boxes, op=op, alpha=1.0, beta=-1.0 if op else -0.1)
    h.use_graphs(True)
    for seed, alpha, beta in ((5, 1.0, 1.0), (5, 2.0, 0.25), (5, 1.0, 1.0), (6, 1.0, 1.0), (6, 0.5, 3.0)):
        h.fill_synthetic(seed, device=True)
        h.set_alpha_beta(alpha, beta)
        got = []
        for mode, bottom in ((0, -1), (1, 0)):
            h.set_bottom_grid(bottom)
            h.set_relax_mode(mode)
            for mixed in (False, True):
                r = h.solve(cmg.solve_params(iter_max=3), mixed=mixed)
                got.append((r["history"].tobytes(), [h.phi(l).tobytes() for l in range(h.nlev)]))
        assert got[:2] == got[2:], (seed, alpha, beta)
    h.set_alpha_beta(1.0, 1.0)
    h.fill_synthetic(5, device=True)
    want = []
    for alpha, beta in ((1.0, 1.0), (2.0, 0.25), (1.0, 1.0)):  # graphs of both kept in between
        h.set_alpha_beta(alpha, beta)
        want.append([h.solve(cmg.solve_params(iter_max=3), mixed=m)["history"].tobytes() for m in (False, True)])
    assert want[0] == want[2] and want[0] != want[1]
    h.close()
