"""The split's iterations on whole warps (sp_ssm_warp_body in
opencaeporo_b200/csrc/flash_phased_kernels.cuh): a short list goes to that
kernel at once, a longer one is finished by it, a long one stays with the
one-lane kernel. A cell's result does not depend on which: 512 fresh cells
flashed alone, as part of 30,000 and as part of 90,000 (6 components: bit for
bit; 9 components, where the compiler rounds the two forms differently: the
parity bar of 1e-8 on the cells whose split converged)."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [6, 9])
def test_result_does_not_depend_on_the_route(nc):
    import torch
    from opencaeporo_b200 import synth
    from opencaeporo_b200.flash import MixtureCompBatch
    from opencaeporo_b200.fluid import synthetic_fluid
    fl = synthetic_fluid(nc, 1234)
    w = synth.uniform_states(fl, 90000, 31)
    got = []
    for n in (512, 30000, 90000):
        m = MixtureCompBatch(fl)
        st = m.new_state(n)
        st.load(w["P"][:n], w["T"][:n], w["Ni"][:n])
        m.flash_fim(st, form="batched", fresh=True)
        torch.cuda.synchronize()
        got.append({k: st.out[k].cpu().numpy()[..., :512] for k in ("phaseNum", "vf", "S", "xij", "iters", "ePEC")})
        m.close()
    for other in got[1:]:
        if nc == 6:
            for k in got[0]:
                np.testing.assert_array_equal(got[0][k], other[k], err_msg=k)
        else:
            np.testing.assert_array_equal(got[0]["phaseNum"], other["phaseNum"])
            ok = (got[0]["ePEC"] <= 1e-9) & (other["ePEC"] <= 1e-9)
            np.testing.assert_allclose(other["vf"][ok], got[0]["vf"][ok], rtol=1e-8)
