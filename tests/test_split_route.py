"""A split's result does not depend on which kernel iterates it. Short lists of
splits go to the whole-warp kernel (sp_ssm_warp_body in
opencaeporo_b200/csrc/flash_phased_kernels.cuh), longer ones to the one-lane
kernel, which may hand its last cells over part-way, and which cells these are
follows the order of atomic appends. Two-phase cells whose warm flash goes
straight to the split (flash type 2: the whole batch is one list) are flashed
in lists of every length class, counted in warps of the whole-warp kernel
(sixteen an SM): every output of a cell is the same, bit for bit, in each, on
repetition and at half the persistent grid, for every component count. Lists
between 3 and 8 cells a warp are the ones that can be handed over."""
import numpy as np
import pytest


def _two_phase(m, fl, n):
    """Inputs and warm-start arrays of n two-phase cells: those of a fresh
    flash, repeated with the pressure moved a little further each time."""
    import torch
    from opencaeporo_b200 import synth
    w = synth.uniform_states(fl, 30000, 31)
    st = m.new_state(30000)
    st.load(w["P"], w["T"], w["Ni"])
    m.flash_fim(st, form="batched", fresh=True)
    torch.cuda.synchronize()
    S = st.out["S"]
    two = torch.nonzero((st.out["phaseNum"] == 3) & (S[0] > 1e-2) & (S[1] > 1e-2)).reshape(-1)
    k = torch.arange(n, device=two.device)
    at, turn = two[k % two.numel()], k // two.numel()
    return {"P": st.P[at] * (1 + 1e-5 * turn), "T": st.T[at], "Ni": st.Ni[:, at],
            "S": S[:, at], "phaseNum": st.out["phaseNum"][at], "xij": st.out["xij"][:, at]}


def _warm(m, inp, n, pct=100):
    import torch
    m.set_tuning(persist_pct=pct)
    st = m.new_state(n)
    for k, v in inp.items():
        dst = getattr(st, k) if k in ("P", "T", "Ni") else st.out[k]
        dst.copy_(v[..., :n])
    m.flash_fim(st, form="batched")
    torch.cuda.synchronize()
    assert (st.out["ftype"] == 2).all()
    return {k: v.cpu().numpy() for k, v in st.out.items()}


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [3, 6, 9, 12])
def test_bits_do_not_depend_on_the_list(nc):
    import torch
    from opencaeporo_b200.flash import MixtureCompBatch
    from opencaeporo_b200.fluid import synthetic_fluid
    fl = synthetic_fluid(nc, 1234)
    m = MixtureCompBatch(fl)
    warps = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    inp = _two_phase(m, fl, 9 * warps)
    want = _warm(m, inp, 9 * warps)
    runs = [(n, 100) for n in (40, warps, 2 * warps, 3 * warps, 3 * warps + 1, 5 * warps, 8 * warps, 8 * warps + 1)]
    for n, pct in runs + [(5 * warps, 100), (5 * warps, 50), (9 * warps, 50)]:
        got = _warm(m, inp, n, pct)
        for k, v in got.items():
            w = want[k][..., :n]
            same = (v == w) | ((v != v) & (w != w)) if v.dtype.kind == "f" else v == w
            assert same.all(), (n, pct, k, np.count_nonzero(~same))
    m.close()
