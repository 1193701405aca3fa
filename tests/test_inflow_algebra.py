"""The algebra of the fast binary64 step (raytracer_3d_gb300/csrc/rt_fast.cu)
restated in numpy and held against the oracle on the CPU: one factor nu per
cell for the mean-flow term and the outgoing upwind fluxes, the inflow V_in*E_in
(from the left neighbour, else the right one, and from the right one too where
two faces converge on the cell), and the limited slopes with H of both faces;
V and H scaled by dt/d where every axis has one spacing, by dt with 1/d per
axis otherwise.  One step from the oracle's state stays within 1e-12 relative
L-infinity of the reference's division form (superbee_fluxes.f90:19-30,
integrate.f90:102-268)."""
import numpy as np
import pytest

from harness import ONX, build_oracle, interior
from test_fast_algebra import CASES, TOL, VEL, _fill_ghosts, _superbee_slope, _take


def inflow_step(o, exp, uniform, h_scale=1.0, converge=True):
    n, dt = exp.n, o.dt
    E = _fill_ghosts(o.E, n, exp.upper, exp.lower)
    e0 = o.E[interior(n)]
    nu = np.zeros(n)
    for c, lam in enumerate(("lambda_x", "lambda_y", "lambda_z")):
        if n[c] > 1:
            nu = nu - dt * getattr(o, lam)[interior(n)]
    acc = np.zeros(n)
    met = 0
    for a in range(6):
        if n[a] <= 1:
            continue
        na = n[a]
        shp = [1] * 6
        shp[a] = na + 1
        df = o.grid["xyzklm"[a]]["dt"][ONX - 1:ONX + na].reshape(shp)      # of faces 0..na
        shp[a] = na
        dc = o.grid["xyzklm"[a]]["dt"][ONX:ONX + na].reshape(shp)          # of the cells
        v = _take(getattr(o, VEL[a]), a, ONX - 1, ONX + na)
        cf = v * dt / df
        V = cf if uniform else v * dt
        H = h_scale * 0.5 * np.abs(V) * (1.0 - np.abs(cf))
        Em1, E0 = _take(E, a, ONX - 2, ONX + na - 1), _take(E, a, ONX - 1, ONX + na)
        Ep1, Ep2 = _take(E, a, ONX, ONX + na + 1), _take(E, a, ONX + 1, ONX + na + 2)
        pos = v > 0
        psi = _superbee_slope(Ep1 - E0, np.where(pos, E0 - Em1, Ep2 - Ep1))
        lo, hi = [slice(None)] * 6, [slice(None)] * 6
        lo[a], hi[a] = slice(0, na), slice(1, na + 1)
        lo, hi = tuple(lo), tuple(hi)
        if not (a == 2 and exp.lower):      # face 0 of an axis whose ghosts copy the edge has no slope
            first = [slice(None)] * 6
            first[a] = slice(0, 1)
            psi[tuple(first)] = 0.0
        vl, vr = v[lo], v[hi]
        nu = nu - (np.maximum(vr, 0.0) - np.minimum(vl, 0.0)) * dt / dc
        inl, inr = vl > 0, vr < 0
        left, right = _take(E, a, ONX - 1, ONX + na - 1), _take(E, a, ONX + 1, ONX + na + 1)
        t = np.where(inl, V[lo] * left, np.where(inr, -V[hi] * right, 0.0))
        if converge:
            t = t + np.where(inl & inr, -V[hi] * right, 0.0)
        met += int(np.count_nonzero(inl & inr))
        t = t + H[lo] * psi[lo] - H[hi] * psi[hi]
        acc = acc + (t if uniform else t / dc)
    return e0 + (e0 * nu + acc), met


def _uniform(o, n):
    return all(np.ptp(o.grid["xyzklm"[a]]["dt"][ONX - 1:ONX + n[a]]) == 0.0 for a in range(6))


@pytest.mark.parametrize("name", list(CASES))
def test_inflow_form_within_bound_of_oracle(name):
    exp = CASES[name]()
    o = build_oracle(exp)
    try:
        forms = (True, False) if _uniform(o, exp.n) else (False,)
        assert (name == "stretched") == (len(forms) == 1)
        for step in range(3):
            got = [inflow_step(o, exp, u) for u in forms]
            wrong = [inflow_step(o, exp, forms[0], h_scale=1.0 + 1e-6)[0],
                     inflow_step(o, exp, forms[0], converge=False)[0]]
            o.integrate(1)
            ref = o.E[interior(exp.n)]
            scale = np.max(np.abs(ref))
            for E, met in got:
                err = np.max(np.abs(E - ref)) / scale
                assert err <= TOL, (step, err)
            # the bound tells a wrong H, and converging faces taken for one, from the right form
            assert np.max(np.abs(wrong[0] - ref)) / scale > TOL
            assert got[0][1] == 0 or np.max(np.abs(wrong[1] - ref)) / scale > TOL
        assert name == "column_1d" or got[0][1] > 0
    finally:
        o.close()
