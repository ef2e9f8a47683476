"""Quotients, reciprocals and square roots on the integer pipe against IEEE arithmetic, and the
exact stepper where a pass item leaves that arithmetic's range (far operands, a gamma at a power of
two), against the oracle: equality of every bit, so no tolerance."""
import ctypes
import dataclasses

import numpy as np
import pytest
import torch

from apophis_gb300 import _capi, hydro, problems
from apophis_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu
SIG = [0, 1, 2, 3, (1 << 52) - 1, (1 << 52) - 2, (1 << 51), (1 << 51) - 1, (1 << 51) + 1, (1 << 29) - 1, 1 << 29]
DIV, RCP, SQRT, MUL = 8, 9, 10, 11


def _values(rng, n, lo, hi):
    """n values of either sign with exponents in lo..hi, a third of them with edge significands."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    edge = rng.integers(0, 3, n) == 0
    m[edge] = np.array(SIG, np.uint64)[rng.integers(0, len(SIG), int(edge.sum()))]
    e = rng.integers(lo + 1023, hi + 1024, n).astype(np.uint64)
    s = rng.integers(0, 2, n).astype(np.uint64)
    return (m | (e << np.uint64(52)) | (s << np.uint64(63))).view(np.float64)


def _run(op, x, y):
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    out = torch.empty_like(xd)
    _capi.call("aph_diag_exact_ops2", op, ctypes.c_void_p(xd.data_ptr()), ctypes.c_void_p(yd.data_ptr()),
               ctypes.c_void_p(out.data_ptr()), x.size, hydro.stream_handle())
    return out.cpu().numpy()


def _same(got, want):
    bad = (got.view(np.uint64) != want.view(np.uint64)) & ~(np.isnan(got) & np.isnan(want))
    assert not bad.any(), (int(bad.sum()), got[bad][:3], want[bad][:3])


@pytest.mark.parametrize("lo,hi", [(-1, 1), (-400, 400), (-405, -395), (395, 405), (-1022, 1023)])
def test_quotients_and_roots_are_ieee(lo, hi):
    rng = np.random.default_rng(10_000 + lo * 7 + hi)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.2e-308, 1.7e308, 1.0, 3.0])
    a, b = (np.concatenate([_values(rng, 400_000, lo, hi), v]) for v in
            (np.repeat(special, special.size), np.tile(special, special.size)))
    # quotients next to representable numbers: b * q rounded, and its neighbours
    q = _values(rng, 100_000, 0, 0)
    c = _values(rng, 100_000, max(lo, -400), min(hi, 400))
    near = np.nextafter(c * q, np.where(rng.integers(0, 2, q.size) == 0, np.inf, -np.inf))
    a, b = np.concatenate([a, near, c * q]), np.concatenate([b, c, c])
    with np.errstate(all="ignore"):
        _same(_run(DIV, a, b), a / b)
        _same(_run(RCP, a, b), 1.0 / b)
        _same(_run(SQRT, a, b), np.sqrt(a))
        r = _values(rng, 100_000, 0, 1)  # roots next to representable numbers
        _same(_run(SQRT, r * r, r), np.sqrt(r * r))


@pytest.mark.parametrize("lo,hi", [(-1, 1), (-205, -195), (195, 205), (-1022, 1023)])
def test_face_products_are_ieee(lo, hi):
    """Products of the fast solvers: rounded as IEEE in their range (zeros included, exponents up to
    the largest and smallest of the operands), refused outside it."""
    rng = np.random.default_rng(20_000 + lo * 7 + hi)
    zero = np.array([0.0, -0.0, 1.0, -3.0, 2.0 ** 900, 2.0 ** -900])
    a, b = (np.concatenate([_values(rng, 400_000, lo, hi), v]) for v in
            (np.repeat(zero, zero.size), np.tile(zero, zero.size)))
    a[:100_000] = 1.0 + rng.integers(0, 1 << 26, 100_000) * 2.0 ** -26  # products half-way between numbers
    b[:100_000] = 1.0 + (2 * rng.integers(0, 1 << 26, 100_000) + 1) * 2.0 ** -27
    with np.errstate(all="ignore"):
        _same(_run(MUL, a, b), a * b)


@pytest.mark.parametrize("recon,rsolver", [("ppm", "hllc"), ("plm", "hlle"), ("ppm", "lhllc"), ("dc", "hllc")])
@pytest.mark.parametrize("gamma,scale", [(2.0, 0), (1.5, 0), (1.0 + 2.0 ** -9, 0), (5.0 / 3.0, -150),
                                         (5.0 / 3.0, 190), (1.4, -260)])
def test_exact_stepper_outside_the_main_path(recon, rsolver, gamma, scale):
    """One RK2 step equals the oracle: gamma at and near powers of two (no small-integer indices),
    densities and energies far from 1 (2^scale: products and quotients beyond the integer pipe's
    range, then windows that are not tame)."""
    from oracle import oracle as O
    cfg, cons = problems.kh2d(n=32, block=16, ng=3, recon=recon, rsolver=rsolver, gamma=gamma)
    cfg = dataclasses.replace(cfg, dfloor=0.0, pfloor=0.0)
    cons = cons * 2.0 ** scale
    ref = O.Mesh(cfg)
    ref.set_cons(cons)
    ref.run(nsteps=2)
    st = Stepper(cfg, cons, exact=True)
    st.step(2)
    sk, sj, si = cfg.interior
    _same(np.ascontiguousarray(st.state()[:, :, sk, sj, si]), np.ascontiguousarray(ref.get()[:, :, sk, sj, si]))
    assert st.status()["dt"] == ref.state()["dt"]
    st.close()


@pytest.mark.parametrize("recon,rsolver", [("ppm", "hllc"), ("ppm", "hlle"), ("ppm", "lhllc"), ("plm", "hlle")])
@pytest.mark.parametrize("scale", [-190, 195, -260, 300])
@pytest.mark.parametrize("path", ["stepper", "driver"])
def test_fast_mode_outside_the_main_path(recon, rsolver, scale, path):
    """Fast mode, densities and energies 2^scale as large (at the edges of tame windows and beyond,
    and products out of range): every operation rounds as before (rsqrt to an ulp), so two steps give
    2^scale times the unscaled ones."""
    cfg, cons = problems.kh2d(n=32, block=16, ng=3, recon=recon, rsolver=rsolver)
    cfg = dataclasses.replace(cfg, dfloor=0.0, pfloor=0.0)
    out = []
    for k in (0, scale):
        if path == "driver":
            dr = hydro.Driver(cfg, cons * 2.0 ** k, exact=False)
            dr.run(nsteps=2)
            got = dr.cons()
        else:
            st = Stepper(cfg, cons * 2.0 ** k, exact=False)
            st.step(2)
            got = st.state()
            st.close()
        sk, sj, si = cfg.interior
        out.append(got[:, :, sk, sj, si] * 2.0 ** -k)
    assert np.allclose(out[1], out[0], rtol=1e-12, atol=1e-13)


@pytest.mark.parametrize("n", [125, 126, 127, 221, 222, 250])
@pytest.mark.parametrize("recon", ["ppm", "plm"])
def test_default_lines_around_the_rule(n, recon):
    """The default lines per item at the widths where their count changes: one step of a single
    block (fewer items than SMs) equals the oracle."""
    from oracle import oracle as O
    cfg, cons = problems.kh2d(n=n, block=n, ng=3, recon=recon, rsolver="hllc")
    ref = O.Mesh(cfg)
    ref.set_cons(cons)
    ref.run(nsteps=1)
    st = Stepper(cfg, cons, exact=True)
    st.step(1)
    sk, sj, si = cfg.interior
    _same(np.ascontiguousarray(st.state()[:, :, sk, sj, si]), np.ascontiguousarray(ref.get()[:, :, sk, sj, si]))
    st.close()


@pytest.mark.parametrize("nx,nscalars", [(159, 0), (160, 0), (161, 0), (321, 0), (1500, 0), (100, 24), (161, 40)])
@pytest.mark.parametrize("recon", ["ppm", "plm"])
def test_flux_segments(nx, nscalars, recon):
    """The per-kernel path's flux kernel cuts long lines (and lines of many scalars) into segments:
    two steps of one long block equal the oracle, exact arithmetic, and the fast ones run."""
    from oracle import oracle as O
    cfg, cons = problems.sod(nx=nx, recon=recon, rsolver="hllc", ng=3)
    if nscalars:
        cfg, cons = problems.with_tracers(cfg, cons, nscalars)
    ref = O.Mesh(cfg)
    ref.set_cons(cons)
    ref.run(nsteps=2)
    sk, sj, si = cfg.interior
    want = ref.get()[:, :, sk, sj, si]
    drv = hydro.Driver(cfg, cons, exact=True)
    drv.run(nsteps=2)
    _same(np.ascontiguousarray(drv.cons()[:, :, sk, sj, si]), np.ascontiguousarray(want))
    fast = hydro.Driver(cfg, cons, exact=False)
    fast.run(nsteps=2)
    assert np.allclose(fast.cons()[:, :, sk, sj, si], want, rtol=1e-10, atol=1e-10)


@pytest.mark.parametrize("recon,rsolver", [("plm", "hlle"), ("plm", "hllc"), ("ppm", "hllc"), ("ppm", "hlle")])
@pytest.mark.parametrize("scale", [-500, 500])
def test_adjoint_outside_the_main_path(recon, rsolver, scale):
    """The adjoint is linear and a power of two changes no rounding: a seed 2^scale as large (products
    beyond the integer pipe's range) gives 2^scale times the gradient, bit for bit."""
    from apophis_gb300.adjoint import Adjoint
    cfg, cons = problems.kh2d_smooth(n=32, block=16, ng=4 if recon == "ppm" else 2, recon=recon,
                                     rsolver=rsolver, integrator="rk2")
    u = torch.from_numpy(cons).cuda()
    lam = torch.zeros_like(u)
    sk, sj, si = cfg.interior
    lam[:, :, sk, sj, si] = torch.randn(lam[:, :, sk, sj, si].shape, dtype=torch.float64, device="cuda",
                                        generator=torch.Generator(device="cuda").manual_seed(11))
    adj = Adjoint(cfg)
    want = adj.step_vjp(u, 2e-3, lam).clone()
    got = adj.step_vjp(u, 2e-3, lam * 2.0 ** scale)
    _same((got * 2.0 ** -scale).cpu().numpy(), want.cpu().numpy())


@pytest.mark.parametrize("n,nscalars,exact", [(126, 30, True), (160, 14, True), (200, 10, True), (221, 12, True),
                                              (221, 12, False)])
def test_default_lines_with_many_scalars(n, nscalars, exact):
    """Widths whose default is two lines per item, with more scalars than two lines leave room for: one
    step equals the oracle (fast mode: it runs)."""
    from oracle import oracle as O
    cfg, cons = problems.kh2d(n=n, block=n, ng=3, recon="ppm", rsolver="hllc")
    cfg, cons = problems.with_tracers(cfg, cons, nscalars)
    st = Stepper(cfg, cons, exact=exact)
    st.step(1)
    sk, sj, si = cfg.interior
    got = np.ascontiguousarray(st.state()[:, :, sk, sj, si])
    st.close()
    ref = O.Mesh(cfg)
    ref.set_cons(cons)
    ref.run(nsteps=1)
    want = np.ascontiguousarray(ref.get()[:, :, sk, sj, si])
    if exact:
        _same(got, want)
    else:
        assert np.allclose(got, want, rtol=1e-10, atol=1e-10)
