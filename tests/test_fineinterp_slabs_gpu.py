"""FineInterp's one-kernel path around its slab height (8 coarse planes per block) and its 16-byte stores: box heights
below, at and above a slab and its multiples, odd widths, on flat arrays aligned to 16 bytes and off by one cell, equal
to the numpy restatement bit for bit."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (3, 5, 7), (8, 8, 8), (5, 4, 9), (16, 12, 15), (7, 16, 16), (13, 3, 17)])
def test_slabs_and_alignment(cmg, nx, ny, nz):
    import torch
    import make_golden_fineinterp as mg
    from test_fineinterp import fine_interp_numpy
    coarse_boxes = sorted((x, y, z, x + 15, y + 15, z + 15) for z in (0, 16) for y in (0, 16) for x in (0, 16))
    # one box inside, one on the domain's low corner, one on its high corner
    lo = [(9, 10, 7), (0, 0, 0), (32 - nx, 32 - ny, 32 - nz)]
    fine_boxes = sorted(tuple(2 * a for a in p) + (2 * (p[0] + nx) - 1, 2 * (p[1] + ny) - 1, 2 * (p[2] + nz) - 1)
                        for p in (lo if nz < 8 else lo[:1]))
    c = mg.seeded_field(coarse_boxes, 32, 80 + nz)
    fi = cmg.FineInterp((0, 0, 0, 63, 63, 63), fine_boxes, coarse_boxes)
    assert fi.is_fused()
    dc = torch.from_numpy(c).cuda()
    for pwc in (False, True):
        want = fine_interp_numpy(coarse_boxes, c, fine_boxes, 32, int(pwc))
        for shift in (0, 1):
            out = torch.full((fi.nfine + 2,), 7.5, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            fi.interp_to_fine_device(dc.data_ptr(), out.data_ptr() + 8 * shift, pwc=pwc)
            torch.cuda.synchronize()
            got = out.cpu().numpy()
            assert np.array_equal(got[shift:shift + fi.nfine], want)
            assert np.all(got[:shift] == 7.5) and np.all(got[shift + fi.nfine:] == 7.5)
    fi.close()
