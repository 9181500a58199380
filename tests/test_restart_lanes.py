"""The restarts on one warp per cell (flash_warp.cuh) against the plain form
over wide ranges of P, T and composition, for every component count: cells
that restart, among them ones whose Rachford-Rice iteration never reaches its
tolerance (all K below one) and ones that reach the restart bound. The two
forms agree to rounding, which a restart chain can amplify: phase counts,
flash types and status are compared, and the phase volumes of the cells both
forms settle."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [3, 6, 9, 12])
def test_restarting_cells_end_as_in_the_plain_form(nc):
    import torch
    from opencaeporo_b200 import synth
    from opencaeporo_b200.flash import MixtureCompBatch
    from opencaeporo_b200.fluid import synthetic_fluid
    fl = synthetic_fluid(nc, 1234 + nc)
    w = synth.uniform_states(fl, 4096, 77 + nc, (2.0, 60.0), (300.0, 450.0), 0.5)
    got = {}
    for form in ("plain", "batched"):
        m = MixtureCompBatch(fl)
        st = m.new_state(4096)
        st.load(w["P"], w["T"], w["Ni"])
        m.flash_fim(st, form=form, fresh=True)
        torch.cuda.synchronize()
        got[form] = st.to_host()
        m.close()
    p, b = got["plain"], got["batched"]
    same = p["phaseNum"] == b["phaseNum"]
    assert (~same).sum() <= 2  # knife-edge cells
    np.testing.assert_array_equal(p["ftype"], b["ftype"])
    settled = same & (p["ePEC"] <= 1e-9) & (b["ePEC"] <= 1e-9)
    np.testing.assert_allclose(b["vf"][settled], p["vf"][settled], rtol=1e-6)
