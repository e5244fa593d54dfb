"""A NaN that the arithmetic makes (infinity minus infinity: its sign bit is set, unlike a NaN from the host) reaches the
residual's max-norm, folded into the residual's pass or not: the solve ends diverged and never reports a norm of the
other cells."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n0,levels,max_box,block,op", [(32, 1, 16, 8, 0), (32, 1, 16, 8, 1), (40, 1, 32, 8, 0),
                                                        (40, 1, 32, 8, 1), (32, 2, 16, 8, 0), (32, 2, 16, 8, 1)])
def test_nan_made_by_the_residual(cmg, n0, levels, max_box, block, op):
    """Boxes of one shape (read across faces), boxes of 32 and 8, and a refined hierarchy; one infinite cell of phi."""
    boxes = (cmg.synthetic_hierarchy(n0, levels, max_box=max_box, seed=3) if levels > 1 else
             [cmg.domain_split((0, 0, 0), (n0 - 1,) * 3, max_box, block)])
    h = cmg.Hierarchy(n0, boxes, op=op, alpha=float(op), beta=-1.0 if op else 1.0)
    h.fill_synthetic(3, device=True)
    phi = [np.zeros(h.num_cells(l)) for l in range(h.nlev)]
    phi[-1][h.num_cells(h.nlev - 1) // 2] = np.inf

    def set_phi():
        for l, p in enumerate(phi):
            h.set_phi(l, p)

    for mode in (0, 1):
        h.set_relax_mode(mode)
        set_phi()
        assert np.isnan(h.residual_norm()) and np.isnan(h.residual_norm_noalloc()), mode
        for mixed in (False, True):
            set_phi()
            r = h.solve(cmg.solve_params(iter_max=2), zero_phi=False, mixed=mixed)
            assert r["diverged"] and r["iterations"] == 0 and np.isnan(r["history"][0]), (mode, mixed)
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("max_box", [16, 32])
def test_nan_in_one_hierarchy_of_a_forest(cmg, max_box):
    """A NaN with the sign bit set in one right-hand side: that hierarchy ends diverged, the others converge."""
    f = cmg.Forest(40, [[cmg.domain_split((0, 0, 0), (39,) * 3, max_box, 8)] for _ in range(3)])
    f.fill_synthetic([1, 2, 3])
    rhs = np.ones(40 ** 3)
    rhs[777] = np.copysign(np.nan, -1.0)
    f.set_rhs(1, 0, rhs)
    for mixed in (False, True):
        r = f.solve(cmg.solve_params(), mixed=mixed)
        assert np.isnan(r[1]["final_norm"]) and r[1]["iterations"] == 0, mixed
        assert all(r[k]["exit_status"] & 1 and r[k]["iterations"] > 0 and r[k]["final_norm"] < 1e-6 for k in (0, 2))
    f.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n0,levels,num_mg", [(32, 1, 1), (32, 2, 1), (24, 3, 2)])
def test_solve_after_a_diverged_one(cmg, n0, levels, num_mg):
    """The V-cycle starts its corrections from zero without clearing them: what a diverged solve left in every field,
    FP64 and FP32, does not reach the next one."""
    boxes = (cmg.synthetic_hierarchy(n0, levels, max_box=16, seed=4) if levels > 1 else
             [cmg.domain_split((0, 0, 0), (n0 - 1,) * 3, 16, 8)])
    h = cmg.Hierarchy(n0, boxes)
    h.fill_synthetic(6, device=True)
    rhs = [h.get_rhs(l) for l in range(h.nlev)]
    p = cmg.solve_params(num_mg=num_mg, iter_max=3)
    for mixed in (False, True):
        want = h.solve(p, mixed=mixed)["history"].tobytes(), [h.phi(l).tobytes() for l in range(h.nlev)]
        h.set_bottom_solver(norm_type=0, small=-1.0)
        for scale in (1e152, 1e153, 1e155, 1e160):  # overflow in the bottom solve's sums, as NaN from there
            for l in range(h.nlev):
                h.set_rhs(l, scale * rhs[l])
            if h.solve(p, mixed=mixed)["diverged"]:
                break
        else:
            pytest.fail("no scale made a NaN")
        h.set_bottom_solver()
        for l in range(h.nlev):
            h.set_rhs(l, rhs[l])
        assert h.solve(p, mixed=mixed)["history"].tobytes() == want[0], mixed
        assert [h.phi(l).tobytes() for l in range(h.nlev)] == want[1], mixed
    h.close()
