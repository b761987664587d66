"""Near-field ptychography (RecNFP) on the GPU against the reference's own
rec_nfp_mpi.py (golden vectors, tests/golden/nfp.npz): synthetic amplitudes,
the objective, the gradient and the Hessian forms at one point, and a
4-iteration BH run (state and step sizes), complex and real projections.
Bound: rel 1e-5 (the BH step sizes 1e-4, as for Rec)."""
import types

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


def nfp_args(n, nobj, ntheta, dt, niter=1):
    return types.SimpleNamespace(
        energy=17.1, detector_pixelsize=3e-6, focustodetectordistance=1.217, z1=8.245e-3,
        ntheta=ntheta, nz=n, n=n, nzobj=nobj, nobj=nobj, obj_dtype=dt, rho=[1, 0.5, 0.1],
        niter=niter, nchunk=ntheta, vis_step=-1, err_step=-1, start_iter=0)


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("tag,dt", [("c", "complex64"), ("f", "float32")])
def test_nfp_cascade_matches_reference(golden, tag, dt):
    from holotomocupy_b200 import RecNFP
    g = golden("nfp")
    n, nobj, ntheta, niter = [int(v) for v in g[f"{tag}_dims"]]
    rec = RecNFP(nfp_args(n, nobj, ntheta, dt))
    truth = {"prb": cuda(g[f"{tag}_prb_true"]), "proj": cuda(g[f"{tag}_proj_true"]), "pos": cuda(g[f"{tag}_pos_true"])}
    rec.gen_sqrt_data(truth, rec.data)
    assert rel_l2(rec.data.cpu().numpy(), g[f"{tag}_data"]) < TOL
    rec.data[:] = cuda(g[f"{tag}_data"])
    V = lambda name: {k: cuda(g[f"{tag}_{name}_{k}"]) for k in ("prb", "proj", "pos")}
    v, gr, et = V("v"), V("g"), V("e")
    assert abs(rec.min(v["prb"], v["proj"], v["pos"]) / float(g[f"{tag}_F"]) - 1) < TOL
    out = {k: torch.zeros_like(x) for k, x in v.items()}
    rec.gradients(v, out)
    for k in ("prb", "proj", "pos"):
        assert rel_l2(out[k].cpu().numpy(), g[f"{tag}_grad_{k}"]) < TOL, k
    assert abs(rec.hessian(v, gr, et) / float(g[f"{tag}_h_ge"]) - 1) < TOL
    assert abs(rec.hessian(v, et, et) / float(g[f"{tag}_h_ee"]) - 1) < TOL


@pytest.mark.parametrize("tag,dt", [("c", "complex64"), ("f", "float32")])
def test_nfp_bh_matches_reference(golden, tag, dt):
    from holotomocupy_b200 import RecNFP
    g = golden("nfp")
    n, nobj, ntheta, niter = [int(v) for v in g[f"{tag}_dims"]]
    rec = RecNFP(nfp_args(n, nobj, ntheta, dt, niter))
    rec.data[:] = cuda(g[f"{tag}_data"])
    rec.vars["prb"][:] = 1
    rec.vars["proj"][:] = 0
    rec.vars["pos"][:] = cuda(g[f"{tag}_pos_true"] + g[f"{tag}_pos_err"])
    record = []
    rec.BH(record=record)
    tb = g[f"{tag}_bh_topbottom"]
    ref_alpha = [tb[0, 0] / tb[0, 1]] + [tb[2 * i, 0] / tb[2 * i, 1] for i in range(1, niter)]
    ref_beta = [0.0] + [tb[2 * i - 1, 0] / tb[2 * i - 1, 1] for i in range(1, niter)]
    for (i, a, b), ra, rb in zip(record, ref_alpha, ref_beta):
        assert abs(a / ra - 1) < 1e-4, (i, a, ra)
        if rb:
            assert abs(b / rb - 1) < 1e-4, (i, b, rb)
    for k in ("prb", "proj", "pos"):
        assert rel_l2(rec.vars[k].cpu().numpy(), g[f"{tag}_bh_{k}"]) < TOL, k


def test_nfp_graph_iteration_matches_host(golden):
    """BH(mode="graph"): step sizes on the device (ht_bh_scalars, ht_axpby_dev)
    and the steady-state iteration replayed from a CUDA graph give the step
    sizes (rtol 1e-9) and the state (rel L2 1e-6) of the host-scalar BH."""
    from holotomocupy_b200 import RecNFP
    g = golden("nfp")
    tag, dt = "c", "complex64"
    n, nobj, ntheta, niter = [int(v) for v in g[f"{tag}_dims"]]
    out = []
    st = torch.cuda.Stream()
    for mode in ("host", "graph"):
        with torch.cuda.stream(st):
            rec = RecNFP(nfp_args(n, nobj, ntheta, dt, niter))
            rec.data[:] = cuda(g[f"{tag}_data"])
            rec.vars["prb"][:] = 1
            rec.vars["proj"][:] = 0
            rec.vars["pos"][:] = cuda(g[f"{tag}_pos_true"] + g[f"{tag}_pos_err"])
            record = []
            rec.BH(record=record, mode=mode)
            out.append((np.array([(a, b) for _, a, b in record]),
                        {k: rec.vars[k].cpu().numpy() for k in ("prb", "proj", "pos")}))
            rec.close()
    (h0, v0), (h1, v1) = out
    assert h1.shape == (niter, 2)
    np.testing.assert_allclose(h1, h0, rtol=1e-9)
    for k in v0:
        assert rel_l2(v1[k], v0[k]) < 1e-6, k


@pytest.mark.parametrize("dt", ["complex64", "float32"])
@pytest.mark.parametrize("nimg", [1, 2, 31, 70, 97])
def test_shared_coefficients_gradient_over_groups(dt, nimg):
    """The gradient of one coefficient array under all images, summed in groups
    whose last one may not be full, against the sum of the gradients of as many
    separate arrays; the other gradients to the bit."""
    import ctypes

    from holotomocupy_b200 import Propagation, _lib
    n, nobj = 32, 48
    rng = np.random.default_rng(nimg)
    real = lambda *s: rng.standard_normal(s).astype("float32")
    c = real(nobj, nobj) if dt == "float32" else (real(nobj, nobj) + 1j * real(nobj, nobj)).astype("complex64")
    c = cuda(0.1 * c)
    prb = cuda((1 + 0.1 * real(1, n, n) + 0.1j * real(1, n, n)).astype("complex64"))
    pos, mag = cuda(4 * real(nimg, 1, 2)), torch.ones(nimg, 1, device="cuda")
    data = cuda(1 + 0.1 * real(nimg, 1, n, n))
    prop = Propagation(n, n, nimg, 1, 7.3e-11, 20e-9, [3e-3])
    out = []
    for shared in (1, 0):
        h = ctypes.c_void_p()
        _lib.call("ht_rec_create", n, n, nobj, nobj, nimg, 1, int(dt == "complex64"), prop._h, ctypes.byref(h))
        _lib.call("ht_rec_set_shared_coefficients", h, shared)
        cs = c if shared else c.expand(nimg, nobj, nobj).contiguous()
        gc, gpos, gprb = torch.empty_like(cs), torch.empty_like(pos), torch.empty_like(prb)
        _lib.call("ht_rec_gradient", h, _lib.ptr(cs), _lib.ptr(pos), _lib.ptr(mag), _lib.ptr(prb), _lib.ptr(data),
                  _lib.ptr(gc), _lib.ptr(gpos), _lib.ptr(gprb), None, 1.0, 1.0, 0, _lib.stream_ptr())
        torch.cuda.synchronize()
        _lib.lib().ht_rec_destroy(h)
        wide = torch.complex128 if gc.is_complex() else torch.float64
        out.append((gc.to(wide) if shared else gc.to(wide).sum(0), gpos, gprb))
    assert rel_l2(out[0][0].cpu().numpy(), out[1][0].cpu().numpy()) < 1e-6
    assert torch.equal(out[0][1], out[1][1]) and torch.equal(out[0][2], out[1][2])
