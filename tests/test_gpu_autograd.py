"""Differentiable operators (holotomocupy_b200.autograd): the backward passes
are the adjoint kernels; checked against the adjoint identity, against
central finite differences of the FP64 oracle, against the reference's own
BH gradient (golden vectors from rec_mpi.py's gradients_cascade) and against
the fused cascade at 256^3 x 360 angles (and 900 angles in chunks).

Bounds: backward vs adjoint kernel rel <= 1e-6 (same kernels); directional
derivatives vs FP64 central differences (step 1e-3 relative) rel <= 1e-4;
gradients vs the reference rel L2 <= 1e-5; autograd vs fused cascade
rel L2 <= 1e-4 (different FP32 summation orders)."""
import types

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import holo_oracle as O

pytestmark = pytest.mark.gpu


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _args(n, ntheta, ndist, niter=1):
    return types.SimpleNamespace(
        energy=17.1, detector_pixelsize=1.4760147601476e-6 * 2 * 2048 / n, focustodetectordistance=1.217,
        z1=(np.array([5.110, 5.464, 6.879, 9.817]) * 1e-3 + 3.135e-3)[:ndist],
        theta=np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32"), ndist=ndist, ntheta=ntheta,
        nz=n, n=n, nzobj=n, nobj=n, obj_dtype="complex64", mask=0.9, lam_prbfit=0.0, rho=[1, 0.05, 0.02],
        niter=niter, nchunk=max(n, ntheta), vis_step=-1, err_step=-1, start_iter=0)


def _redot(a, b):
    a, b = a.to(torch.complex128), b.to(torch.complex128)
    return float(torch.sum(a.real * b.real + a.imag * b.imag))


def test_linear_backwards_are_the_adjoints():
    from holotomocupy_b200 import Propagation, Tomo
    from holotomocupy_b200.autograd import propagate, radon
    g = torch.Generator(device="cuda").manual_seed(3)
    cn = lambda *s: torch.randn(*s, dtype=torch.complex64, device="cuda", generator=g)
    n = 64
    tomo = Tomo(n, n, np.linspace(0, np.pi, 20, endpoint=False).astype("float32"), 0)
    x = cn(n, n, n).requires_grad_()
    w = cn(20, n, n)
    y = radon(x, tomo)
    (gx,) = torch.autograd.grad(_redot_t(y, w), x)
    assert rel_l2(gx.cpu().numpy(), tomo.RT(w).cpu().numpy()) < 1e-6
    prop = Propagation(n, n, 3, 2, 7.3e-11, 20e-9, [3e-3, 5e-3])
    x = cn(3, n, n).requires_grad_()
    w = cn(3, n, n)
    (gx,) = torch.autograd.grad(_redot_t(propagate(x, 1, prop), w), x)
    assert rel_l2(gx.cpu().numpy(), prop.DT(w, 1).cpu().numpy()) < 1e-6


def _redot_t(a, b):
    return torch.sum(a.real * b.real + a.imag * b.imag)


def test_shift_derivatives_against_fp64_central_differences():
    """d/dh Re<S(coeff(psi + h dpsi); pos + h dpos), w> from the backward pass
    against central differences of the FP64 oracle's curlyS."""
    from holotomocupy_b200 import Shift
    from holotomocupy_b200.autograd import shift
    n, B = 64, 6
    rng = np.random.default_rng(5)
    cn = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s))
    psi = cn(B, n, n).astype("complex64")
    pos = rng.uniform(-3, 3, (B, 2)).astype("float32")
    mag = rng.uniform(0.9, 1.1, B).astype("float32")
    w = cn(B, n, n).astype("complex64")
    dpsi = cn(B, n, n).astype("complex64")
    dpos = rng.uniform(-1, 1, (B, 2)).astype("float32")
    sh = Shift(n, n, n, n, "complex64")
    tp, tq = cuda(psi).requires_grad_(), cuda(pos).requires_grad_()
    out = shift(tp, tq, cuda(mag), sh)
    gp, gq = torch.autograd.grad(_redot_t(out, cuda(w)), (tp, tq))
    osh = O.Shift(n, n, n, n, "complex64", dtype="complex128")
    f = lambda p, q: float(np.sum((np.conj(w.astype(np.complex128)) * osh.curlyS(p, q, mag.astype(np.float64))).real))
    for name, (d_psi, d_pos) in {"psi": (dpsi, 0 * dpos), "pos": (0 * dpsi, dpos)}.items():
        scale = np.linalg.norm(psi) / np.linalg.norm(d_psi) if name == "psi" else \
            np.linalg.norm(pos) / np.linalg.norm(d_pos)
        h = 1e-3 * scale
        p0, q0 = psi.astype(np.complex128), pos.astype(np.float64)
        fd = (f(p0 + h * d_psi, q0 + h * d_pos) - f(p0 - h * d_psi, q0 - h * d_pos)) / (2 * h)
        an = _redot(gp, cuda(d_psi)) + float(torch.sum(gq.double() * cuda(d_pos).double()))
        assert abs(an / fd - 1) < 1e-4, (name, an, fd)


def _golden_setup(g):
    from holotomocupy_b200.autograd import DataFidelity
    from holotomocupy_b200.rec import Rec
    n, ntheta, ndist, nobj = [int(v) for v in g["c_dims"]]
    rec = Rec(_args(n, ntheta, ndist))
    mag = (1 + rec.shrink_nd) / cuda(rec.norm_magnifications[None, :].astype("float32"))
    return rec, DataFidelity.from_rec(rec), mag.contiguous()


@pytest.mark.parametrize("chunk", [None, 4])
def test_fidelity_gradient_matches_reference_bh_gradient(golden, chunk):
    """Autograd through R-free data term (variable proj) against the
    reference's gradients_cascade on the same inputs (golden vectors)."""
    from holotomocupy_b200.autograd import DataFidelity
    g = golden("rec")
    rec, fid, mag = _golden_setup(g)
    if chunk:
        fid = DataFidelity.from_rec(rec, chunk=chunk)
    prb = cuda(g["c_prb"]).requires_grad_()
    proj = cuda(g["c_proj"]).requires_grad_()
    pos = cuda(g["c_pos"]).requires_grad_()
    F = fid(proj, prb, pos, mag, cuda(g["c_data"]), proj=True)
    assert abs(F.item() / float(g["c_F"]) - 1) < 1e-5
    gprb, gproj, gpos = torch.autograd.grad(F, (prb, proj, pos))
    r = rec.rho_sq
    assert rel_l2((gprb * r["prb"]).cpu().numpy(), g["c_grad_prb"]) < 1e-5
    assert rel_l2((gproj * r["obj"]).cpu().numpy(), g["c_grad_proj"]) < 1e-5
    assert rel_l2((gpos * r["pos"]).cpu().numpy(), g["c_grad_pos"]) < 1e-5


def test_fidelity_directional_derivative_against_fp64_central_differences():
    from holotomocupy_b200.autograd import DataFidelity
    from holotomocupy_b200.rec import Rec
    n, ntheta, ndist = 64, 8, 2
    args = _args(n, ntheta, ndist)
    rec = Rec(args)
    orc = O.Rec(args, "complex128")
    rng = np.random.default_rng(11)
    mag = rng.uniform(0.95, 1.05, (ntheta, ndist)).astype("float32")
    orc.eff_demagnifications[:] = mag
    cn = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    x = {"prb": (1 + 0.1 * cn(ndist, n, n)).astype("complex64"), "proj": (0.05 * cn(ntheta, n, n)).astype("complex64"),
         "pos": rng.uniform(-3, 3, (ntheta, ndist, 2)).astype("float32")}
    v = {"prb": cn(ndist, n, n).astype("complex64"), "proj": cn(ntheta, n, n).astype("complex64"),
         "pos": rng.uniform(-1, 1, (ntheta, ndist, 2)).astype("float32")}
    data = (np.abs(rng.standard_normal((ntheta, ndist, n, n))) + 0.5).astype("float32")
    fid = DataFidelity.from_rec(rec)
    t = {k: cuda(a).requires_grad_() for k, a in x.items()}
    F = fid(t["proj"], t["prb"], t["pos"], cuda(mag), cuda(data), proj=True)
    gr = dict(zip(("prb", "proj", "pos"), torch.autograd.grad(F, (t["prb"], t["proj"], t["pos"]))))
    d64 = data.astype(np.float64)
    f = lambda y: orc.F0(orc.F1(orc.F2(orc.F3([y["prb"], y["proj"], y["pos"]]))), d64)
    for k in ("prb", "proj", "pos"):
        h = 1e-3 * np.linalg.norm(x[k]) / np.linalg.norm(v[k])
        up = {kk: a.astype(np.complex128 if np.iscomplexobj(a) else np.float64) for kk, a in x.items()}
        dn = dict(up)
        up[k] = up[k] + h * v[k]
        dn[k] = dn[k] - h * v[k]
        fd = (f(up) - f(dn)) / (2 * h)
        an = _redot(gr[k], cuda(v[k])) if k != "pos" else float(torch.sum(gr[k].double() * cuda(v[k]).double()))
        assert abs(an / fd - 1) < 1e-4, (k, an, fd)


def _phantom_problem(n, ntheta, ndist, pos_amp, seed):
    from holotomocupy_b200 import synthetic
    from holotomocupy_b200.rec import Rec
    args = _args(n, ntheta, ndist)
    rec = Rec(args)
    obj = synthetic.ellipsoid_phantom(n, 20, seed)
    prb = synthetic.random_probe(ndist, n, n, seed + 1)
    pos = synthetic.random_positions(ntheta, ndist, pos_amp, seed + 2)
    rec.eff_demagnifications[:] = (1 + rec.shrink_nd) / cuda(rec.norm_magnifications[None, :].astype("float32"))
    g = torch.Generator(device="cuda").manual_seed(seed + 4)
    # phases of ~0.1 rad (100x the phantom's) so that the object term weighs in
    rec.data.copy_(rec.forward_amplitudes(100 * obj, prb, pos))
    x = {"obj": 90 * obj, "prb": torch.ones_like(prb),
         "pos": pos + 0.5 * (2 * torch.rand(pos.shape, generator=g, device="cuda") - 1)}
    synthetic.noisy_amplitudes(rec.data, 1e4, seed + 3)
    return rec, x, rec.data


@pytest.mark.parametrize("ntheta,chunk", [(360, None), (360, 90), (900, 225)])
def test_autograd_matches_fused_cascade_at_256(ntheta, chunk):
    """256^3 object, 4 distances, 256^2 detector, positions +-3 px: the
    composed autograd gradient (object variable, through R) equals the fused
    cascade's (Rec.gradients), with and without angle-chunk recomputation."""
    from holotomocupy_b200.autograd import DataFidelity
    n, ndist = 256, 4
    rec, x, data = _phantom_problem(n, ntheta, ndist, 3.0, 31)
    vars = {"obj": x["obj"], "prb": x["prb"], "pos": x["pos"], "proj": rec.fwd_tomo(x["obj"])}
    grads = {k: torch.zeros_like(v) for k, v in vars.items()}
    rec.gradients(vars, grads)
    fid = DataFidelity.from_rec(rec, chunk=chunk)
    t = {k: x[k].clone().requires_grad_() for k in ("obj", "prb", "pos")}
    F = fid(t["obj"], t["prb"], t["pos"], rec.eff_demagnifications, data)
    gobj, gprb, gpos = torch.autograd.grad(F, (t["obj"], t["prb"], t["pos"]))
    r = rec.rho_sq
    assert rel_l2((gprb * r["prb"]).cpu().numpy(), grads["prb"].cpu().numpy()) < 1e-4
    assert rel_l2((gpos * r["pos"]).cpu().numpy(), grads["pos"].cpu().numpy()) < 1e-4
    assert rel_l2((gobj * r["obj"]).cpu().numpy(), grads["obj"].cpu().numpy()) < 1e-4


@pytest.mark.parametrize("n,nobj,obj_dtype,chunk", [(32, 48, "complex64", None), (64, 64, "complex64", 3),
                                                    (64, 96, "float32", 4), (128, 256, "complex64", 5)])
@pytest.mark.parametrize("proj", [False, True])
def test_fidelity_fused_equals_operator_by_operator(n, nobj, obj_dtype, chunk, proj):
    """The fused term against the composition of the single operators (which a
    data gradient asks for): value and gradients, ragged chunks, object wider
    than the detector, a distance whose probe is zero (|x0| has gradient 0 there)."""
    from holotomocupy_b200.autograd import DataFidelity
    rng = np.random.default_rng(n + nobj)
    ntheta, ndist, nz = 7, 2, 64
    theta = np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")
    fid = DataFidelity.create(n, nz, nobj, nobj, theta, ndist, 7.3e-11, 20e-9, np.array([3e-3, 5e-3]), 0.9, chunk,
                              obj_dtype)
    shape = (ntheta, nobj, nobj) if proj else (nobj, nobj, nobj)
    x = 0.05 * rng.standard_normal(shape).astype("float32")
    if obj_dtype == "complex64":
        x = (x + 0.01j * rng.standard_normal(shape)).astype("complex64")
    prb = (1 + 0.1 * rng.standard_normal((ndist, nz, n)) + 0.1j).astype("complex64")
    prb[1] = 0
    pos = rng.uniform(-3, 3, (ntheta, ndist, 2)).astype("float32")
    mag = rng.uniform(0.9, 1.0, (ntheta, ndist)).astype("float32")
    data = (1 + 0.1 * rng.standard_normal((ntheta, ndist, nz, n))).astype("float32")
    res = []
    for fused in (True, False):
        t = [cuda(a).requires_grad_() for a in (x, prb, pos)]
        d = cuda(data).requires_grad_(not fused)
        assert fid._use_fused(t[0], t[1], t[2], cuda(mag), d, proj) == fused
        f = fid(*t, cuda(mag), d, proj=proj)
        res.append([f.detach()] + list(torch.autograd.grad(2 * f, t)))
    for a, b in zip(*res):
        assert a.dtype == b.dtype and a.shape == b.shape
        assert torch.isfinite(torch.view_as_real(a) if a.is_complex() else a).all()
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-5, rel_l2(a.cpu().numpy(), b.cpu().numpy())


def _small_fidelity(seed=5, n=32, ntheta=5, ndist=2, chunk=None, obj_dtype="complex64"):
    """A data term the fused cascade takes, and its inputs (obj, prb, pos, mag, data)."""
    from holotomocupy_b200.autograd import DataFidelity
    rng = np.random.default_rng(seed)
    theta = np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")
    fid = DataFidelity.create(n, n, n, n, theta, ndist, 7.3e-11, 20e-9, np.linspace(3e-3, 5e-3, ndist), 0.9, chunk,
                              obj_dtype)
    obj = (0.05 * rng.standard_normal((n, n, n))).astype(obj_dtype)
    prb = (1 + 0.1 * rng.standard_normal((ndist, n, n)) + 0.1j).astype("complex64")
    pos = rng.uniform(-3, 3, (ntheta, ndist, 2)).astype("float32")
    mag = rng.uniform(0.9, 1.0, (ntheta, ndist)).astype("float32")
    data = (1 + 0.1 * rng.standard_normal((ntheta, ndist, n, n))).astype("float32")
    return fid, [cuda(a) for a in (obj, prb, pos, mag, data)]


def test_fidelity_follows_its_operators_settings():
    """The propagator set to the padded grid, or one of another size or of a type
    of its own in its place: operator by operator, as the operators themselves go."""
    from holotomocupy_b200 import Propagation

    class Half(Propagation):
        def D(self, psi, j):
            return 0.5 * super().D(psi, j)
    fid, args = _small_fidelity()
    ref = fid(*args)
    calls = []
    padded = fid.prop._padded
    fid.prop._padded = lambda *a: calls.append(a[1]) or padded(*a)
    fid.prop._use_cufftdx = False
    assert not fid._use_fused(*args, False)
    assert rel_l2(fid(*args).cpu().numpy(), ref.cpu().numpy()) < 1e-5
    assert calls == [0, 1]
    fid.prop = Propagation(32, 32, 5, 3, 7.3e-11, 20e-9, [3e-3, 5e-3, 9e-3])
    assert not fid._use_fused(*args, False)
    assert rel_l2(fid(*args).cpu().numpy(), ref.cpu().numpy()) < 1e-5
    fid.prop = Half(32, 32, 5, 2, 7.3e-11, 20e-9, [3e-3, 5e-3])
    assert not fid._use_fused(*args, False)
    assert abs(fid(*args) - 0.25) < 0.05   # amplitudes near 1/2 under data near 1


def _value_and_grads(fid, args, proj=False):
    t = [a.clone().requires_grad_() for a in args[:3]]
    f = fid(*t, *args[3:], proj=proj)
    return [f.detach()] + list(torch.autograd.grad(f, t))


def test_fidelity_takes_a_replaced_propagator():
    """A propagator put in the place of the first one is the one that counts, also
    after the first is gone and its tables' memory is in other hands, and a
    backward pass keeps the operators its forward pass had."""
    from holotomocupy_b200 import Propagation
    fid, args = _small_fidelity()
    first = _value_and_grads(fid, args)
    t = [a.clone().requires_grad_() for a in args[:3]]
    f = fid(*t, *args[3:])
    fid.prop = Propagation(32, 32, 5, 2, 7.3e-11, 20e-9, [9e-3, 12e-3])
    got = _value_and_grads(fid, args)
    other, _ = _small_fidelity()
    other.prop = fid.prop
    other._use_fused = lambda *a: False
    for a, b in zip(got, _value_and_grads(other, args)):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-5
    assert abs(got[0] - first[0]) > 1e-3 * first[0]
    for a, b in zip(torch.autograd.grad(f, t), first[1:]):
        assert torch.equal(a, b)


def test_fidelity_holds_no_memory_between_calls():
    """The cascade's workspaces come from torch's allocator and go back with the
    call, ragged chunks and several streams included: after a call nothing is
    held, inside torch or outside."""
    fid, args = _small_fidelity(n=64, ntheta=7, chunk=4)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()):
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            _value_and_grads(fid, args)
        torch.cuda.synchronize()
    held, free = torch.cuda.memory_allocated(), torch.cuda.mem_get_info()[0] + torch.cuda.memory_reserved()
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            _value_and_grads(fid, args)
        torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() == held
    assert torch.cuda.mem_get_info()[0] + torch.cuda.memory_reserved() == free


@pytest.mark.parametrize("n,ntheta,ndist,chunk", [(64, 45, 2, None), (64, 46, 4, 23)])
def test_fidelity_peak_memory_is_that_of_the_operators(n, ntheta, ndist, chunk):
    """Peak of a value, and of a value with gradients, over the inputs: the fused
    cascade's at most that of the composition and a tenth."""
    peaks = {}
    for fused in (True, False):
        fid, args = _small_fidelity(n=n, ntheta=ntheta, ndist=ndist, chunk=chunk)
        if not fused:
            fid._use_fused = lambda *a: False
        for grads in (False, True):
            run = (lambda: _value_and_grads(fid, args)) if grads else (lambda: fid(*args))
            run()
            torch.cuda.synchronize()
            torch.cuda.reset_peak_memory_stats()
            base = torch.cuda.memory_allocated()
            run()
            peaks[fused, grads] = torch.cuda.max_memory_allocated() - base
    assert peaks[True, False] <= 1.1 * peaks[False, False], peaks
    assert peaks[True, True] <= 1.1 * peaks[False, True], peaks


def test_fidelity_under_capture():
    """Value and gradients recorded into a graph and replayed on other inputs."""
    fid, args = _small_fidelity(chunk=3)
    _, other = _small_fidelity(seed=6, chunk=3)
    ref = _value_and_grads(fid, other)
    bufs = [a.clone() for a in args]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        _value_and_grads(fid, bufs)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _value_and_grads(fid, bufs)
    for b, o in zip(bufs, other):
        b.copy_(o)
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, ref):
        assert torch.equal(a, b)


def test_fidelity_from_two_threads():
    """Two data terms of one shift and one propagator, each in a thread and on a
    stream of its own: the values and gradients of one after the other."""
    import threading

    from holotomocupy_b200.autograd import DataFidelity
    fid, args = _small_fidelity(n=64, ntheta=6, chunk=4)
    fids = [fid, DataFidelity(fid.sh, fid.prop, np.linspace(0, np.pi, 6, endpoint=False), 0.9, 64, 64, 4)]
    sets = [args, _small_fidelity(seed=8, n=64, ntheta=6, chunk=4)[1]]
    refs = [_value_and_grads(f, a) for f, a in zip(fids, sets)]
    torch.cuda.synchronize()
    res, errors = [None, None], []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    res[i] = _value_and_grads(fids[i], sets[i])
                torch.cuda.current_stream().synchronize()
        except Exception as e:   # shown by the assertion below
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for got, ref in zip(res, refs):
        for a, b in zip(got, ref):
            assert torch.equal(a, b)


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("wrt", [0, 1, 2])
def test_second_derivatives_are_refused(fused, wrt):
    """A derivative of the data term's gradients, whose main terms autograd cannot
    see, raises instead of giving the rest."""
    fid, args = _small_fidelity(n=32, ntheta=3)
    if not fused:
        fid._use_fused = lambda *a: False
    t = [a.clone().requires_grad_() for a in args[:3]]
    f = fid(*t, *args[3:])
    g = torch.autograd.grad(f ** 2, t, create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        (f + g[wrt].abs().sum()).backward()


@pytest.mark.parametrize("far", [float("inf"), -float("inf"), 1e30, -1e30, 4000.0, -33.0])
@pytest.mark.parametrize("axis", [0, 1])
def test_fidelity_of_an_image_far_off_the_object(far, axis):
    """An image shifted off the object, infinitely far included, sees its zeros: the
    fused term's value and gradients against the composition's."""
    fid, args = _small_fidelity()
    args[2][1, 0, axis] = far
    fused = _value_and_grads(fid, args)
    assert fid._use_fused(*args, False)
    fid._use_fused = lambda *a: False
    for a, b in zip(fused, _value_and_grads(fid, args)):
        assert torch.isfinite(torch.view_as_real(a) if a.is_complex() else a).all()
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-5


@pytest.mark.parametrize("mag", [1e4, -1e7, 1e30, float("inf"), -float("inf")])
def test_fidelity_of_an_image_magnified_off_the_object(mag):
    """At a magnification that puts every pixel off the object, infinite included,
    an image sees its zeros: fused against composed."""
    fid, args = _small_fidelity()
    args[3][2, 1] = mag
    fused = _value_and_grads(fid, args)
    assert fid._use_fused(*args, False)
    fid._use_fused = lambda *a: False
    for a, b in zip(fused, _value_and_grads(fid, args)):
        assert torch.isfinite(torch.view_as_real(a) if a.is_complex() else a).all()
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-5


@pytest.mark.parametrize("proj", [False, True])
def test_fidelity_under_saved_tensor_hooks(proj):
    """Saved tensors kept on the host, and ones that come back with other strides:
    the gradients without hooks, to the bit."""
    fid, args = _small_fidelity(chunk=3)
    if proj:
        args[0] = torch.cat([t.R(args[0]) for t in fid.tomos])
    ref = _value_and_grads(fid, args, proj)
    strided = lambda t: torch.stack([t, t], -1)[..., 0]
    for hooks in (torch.autograd.graph.save_on_cpu(pin_memory=True),
                  torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: strided(t.cuda()))):
        with hooks:
            got = _value_and_grads(fid, args, proj)
        for a, b in zip(got, ref):
            assert torch.equal(a, b)
