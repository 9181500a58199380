"""ocpf_fim_jacobian at the edges of its connection tiles (32 connections a
warp, at most five rows a thread) for every component count, against the
restatement bit for bit: mixed one- and two-phase bulks, phases absent
upstream, zero mole fractions, viscosities and densities whose quotients
leave the shared-reciprocal range, and a phase whose composition count
differs between the two ends."""
import numpy as np
import pytest

from oracle import fim_jacobian as J


def _bulk(nc, n, seed):
    rng = np.random.default_rng(seed)
    ncom, ncol = nc + 1, nc + 2
    kind = rng.integers(0, 3, n)  # 0 oil, 1 gas, 2 both
    ex = np.stack([kind != 1, kind != 0, np.ones(n, bool)], axis=1).astype(np.int64)
    vn = ex * np.array([nc, nc, 0])
    # one phase short of a composition at some two-phase bulks: its columns
    # at the other end run into the next phase's
    short = (kind == 2) & (rng.uniform(size=n) < 0.2)
    vn[short, 0] -= 1
    x = rng.dirichlet(np.ones(ncom), (n, 3))
    x[:, :2, nc] = 0
    x[rng.uniform(size=n) < 0.2, 0, 0] = 0
    u = lambda lo, hi, *s: rng.uniform(lo, hi, s)  # noqa: E731
    part = lambda: rng.normal(size=(n, 3, ncom)) * (rng.uniform(size=(n, 3, ncom)) < 0.9)  # noqa: E731
    mu = u(0.02, 1.0, n, 3)
    xi = u(0.2, 3.0, n, 3)
    far = rng.uniform(size=n) < 0.1
    mu[far, 0] *= 1e-70
    xi[rng.uniform(size=n) < 0.1, 1] *= 1e-90
    S = rng.dirichlet(np.ones(3), n) * ex
    return {"phaseExist": ex, "pSderExist": ex, "pVnumCom": vn, "S": S, "rho": u(5, 60, n, 3), "xi": xi, "mu": mu,
            "muP": u(1e-6, 1e-5, n, 3), "xiP": u(1e-6, 1e-5, n, 3), "rhoP": u(1e-5, 1e-4, n, 3), "xij": x,
            "rhox": part(), "xix": part(), "mux": part(), "dSec_dPri": rng.normal(size=(n, 3 * ncol * ncol)),
            "vfP": -u(0.01, 0.2, n), "vfi": u(0.3, 5, n, ncom), "kr": u(0, 1, n, 3) * (u(0, 1, n, 3) < 0.9),
            "Pj": u(2990, 3010, n, 3), "dKr_dS": rng.normal(size=(n, 3, 3)), "dPcj_dS": rng.normal(size=(n, 3, 3)),
            "v": u(500, 1500, n), "poroP": u(1e-7, 1e-6, n), "depth": u(8000, 8010, n)}


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [3, 6, 9, 12])
@pytest.mark.parametrize("nconn", [1, 31, 33, 97])
def test_tile_edges_match_restatement_bit_for_bit(nc, nconn):
    import torch
    from opencaeporo_b200.fim_jacobian import ConnGraph
    from test_fim_jacobian import _soa
    n, ncom, ncol = 40, nc + 1, nc + 2
    bk = _bulk(nc, n, 100 * nc + nconn)
    rng = np.random.default_rng(nconn)
    b = rng.integers(0, n, nconn)
    e = (b + 1 + rng.integers(0, n - 1, nconn)) % n
    cn = {"bId": b.astype(np.int64), "eId": e.astype(np.int64), "area": rng.uniform(1, 100, nconn)}
    g = ConnGraph(n, cn["bId"], cn["eId"], cn["area"])
    dbk = _soa({k: np.asarray(v).reshape(n, -1) if np.ndim(v) > 1 else v for k, v in bk.items()}, n)
    up, rho = g.upwind(dbk)
    out = g.jacobian(nc, 0.25, dbk, up, rho)
    torch.cuda.synchronize()
    g.close()
    cn["upblock"], cn["upblock_Rho"] = J.upwind(bk, cn)
    want = J.assemble(bk, cn, ncom, 0.25)
    np.testing.assert_array_equal(up.cpu().numpy().T, cn["upblock"])
    for k, w in zip(("diag", "offEB", "offBE"), want):
        np.testing.assert_array_equal(out[k].cpu().numpy().T.reshape(-1, ncol, ncol), w, err_msg=k)
