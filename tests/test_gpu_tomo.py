"""USFFT Radon transform on the GPU against the reference (golden vectors from
its own tomo.py) and the oracle.  Bound: rel L2 <= 1e-5 against the reference
and the FP32 oracle; the FP64 oracle is reported with a 1e-4 bound."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import holo_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("tag", ["a", "b", "c"])
def test_R_RT_match_reference(golden, tag):
    from holotomocupy_b200 import Tomo
    g = golden("tomo")
    n, nz = int(g[f"{tag}_n"]), int(g[f"{tag}_nz"])
    t = Tomo(n, nz, g[f"{tag}_theta"], float(g[f"{tag}_mask_r"]))
    assert t.pars[0] == int(g[f"{tag}_m"])
    np.testing.assert_array_equal(t.pars[2].cpu().numpy(), g[f"{tag}_phi"])
    for src, op, key in [("xc", t.R, "Rxc"), ("yc", t.RT, "RTyc"), ("xf", t.R, "Rxf"), ("yf", t.RT, "RTyf")]:
        out = op(torch.from_numpy(g[f"{tag}_{src}"]).cuda()).cpu().numpy()
        ref = g[f"{tag}_{key}"]
        assert out.shape == ref.shape and out.dtype == ref.dtype
        assert rel_l2(out, ref) < TOL, (key, rel_l2(out, ref))


@pytest.mark.parametrize("n,ntheta,nz", [(128, 180, 3), (256, 96, 2), (384, 48, 2), (512, 32, 2)])
def test_R_RT_against_oracle(n, ntheta, nz):
    from holotomocupy_b200 import Tomo
    rng = np.random.default_rng(n)
    theta = np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")
    t = Tomo(n, nz, theta, 0.9)
    o32 = O.Tomo(n, nz, theta, 0.9, "complex64")
    o64 = O.Tomo(n, nz, theta, 0.9, "complex128")
    x = (rng.standard_normal((nz, n, n)) + 1j * rng.standard_normal((nz, n, n))).astype("complex64")
    y = (rng.standard_normal((ntheta, nz, n)) + 1j * rng.standard_normal((ntheta, nz, n))).astype("complex64")
    Rx = t.R(torch.from_numpy(x).cuda()).cpu().numpy()
    RTy = t.RT(torch.from_numpy(y).cuda()).cpu().numpy()
    assert rel_l2(Rx, o32.R(x)) < TOL
    assert rel_l2(RTy, o32.RT(y)) < TOL
    assert rel_l2(Rx, o64.R(x.astype(np.complex128))) < 1e-4
    assert rel_l2(RTy, o64.RT(y.astype(np.complex128))) < 1e-4


def test_adjoint_float32():
    """tests/tomo/test_tomo.ipynb cell 15 of the reference, asserted."""
    from holotomocupy_b200 import Tomo
    n, nz, ntheta = 256, 16, 1024
    theta = np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")
    t = Tomo(n, nz, theta, 1)
    rng = np.random.default_rng(42)
    x = torch.from_numpy(rng.standard_normal((nz, n, n)).astype("float32")).cuda()
    y = torch.from_numpy(rng.standard_normal((ntheta, nz, n)).astype("float32")).cuda()
    Rx, RTy = t.R(x), t.RT(y)
    assert Rx.dtype == torch.float32 and tuple(Rx.shape) == (ntheta, nz, n)
    lhs = torch.sum(Rx.double() * y.double()).item()
    rhs = torch.sum(x.double() * RTy.double()).item()
    assert abs(lhs - rhs) / abs(lhs) < 1e-5


def test_fbp_matches_oracle():
    from holotomocupy_b200 import Tomo
    n, nz, ntheta = 64, 2, 96
    theta = np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")
    rng = np.random.default_rng(3)
    d = rng.standard_normal((ntheta, nz, n)).astype("float32")
    t = Tomo(n, nz, theta, 1)
    o = O.Tomo(n, nz, theta, 1, "complex128")
    for f in ("ramp", "shepp", "parzen"):
        got = t.fbp(torch.from_numpy(d).cuda(), f).cpu().numpy()
        assert rel_l2(got, o.fbp(d.astype(np.float64), f)) < 1e-5
    with pytest.raises(ValueError):
        t.fbp(torch.from_numpy(d).cuda(), "hann")


def test_slice_capacity_is_enforced():
    """The library refuses more slices than the handle's workspace holds; the
    Python class then runs taller volumes slab by slab, and refuses wrong
    shapes."""
    from holotomocupy_b200 import Tomo, _lib
    t = Tomo(32, 2, np.linspace(0, np.pi, 8, endpoint=False), 0)
    x = torch.zeros(3, 32, 32, dtype=torch.complex64, device="cuda")
    y = torch.empty(8, 3, 32, dtype=torch.complex64, device="cuda")
    assert _lib.lib().ht_tomo_R(t._h, _lib.ptr(x), _lib.ptr(y), 3, _lib.stream_ptr()) == 1
    assert tuple(t.R(x).shape) == (8, 3, 32)
    with pytest.raises(ValueError):
        t.R(torch.zeros(3, 32, 31, dtype=torch.complex64, device="cuda"))


@pytest.mark.parametrize("n,ntheta,nz", [(64, 40, 24), (128, 90, 32)])
def test_prefilter_folded_into_R_and_RT(n, ntheta, nz):
    """coeff(R obj) = Cx R Cz obj and R^T coeff(sino) = Cz R^T Cx sino, with Cx
    applied inside R's detector spectrum (ht_tomo_R_coeffx / ht_tomo_RT_coeffx)
    and Cz on the volume (ht_shift_coeff_z): the BH iteration's form."""
    from holotomocupy_b200 import Shift, Tomo, _lib
    rng = np.random.default_rng(n + 1)
    theta = np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")
    t = Tomo(n, nz, theta, 0.9)
    sh = Shift(n, n, nz, nz, "complex64")
    cn = lambda *s: torch.from_numpy((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype("complex64")).cuda()
    x, y = cn(nz, n, n), cn(ntheta, nz, n)
    st = _lib.stream_ptr()
    # forward
    ref = sh.coeff(t.R(x))
    xz = x.clone()
    _lib.call("ht_shift_coeff_z", sh._hc, _lib.ptr(xz), _lib.ptr(xz), n * n, st)
    got = torch.empty(ntheta, nz, n, dtype=torch.complex64, device="cuda")
    _lib.call("ht_tomo_R_coeffx", t._h, _lib.ptr(xz), _lib.ptr(got), nz, st)
    assert rel_l2(got.cpu().numpy(), ref.cpu().numpy()) < 1e-5
    # adjoint
    ref = t.RT(sh.coeff(y))
    got = torch.empty(nz, n, n, dtype=torch.complex64, device="cuda")
    _lib.call("ht_tomo_RT_coeffx", t._h, _lib.ptr(y), _lib.ptr(got), nz, 1.0, st)
    _lib.call("ht_shift_coeff_z", sh._hc, _lib.ptr(got), _lib.ptr(got), n * n, st)
    assert rel_l2(got.cpu().numpy(), ref.cpu().numpy()) < 1e-5
    # the scaled adjoint and the out-of-place z prefilter (the BH gradient's form)
    scaled = torch.empty_like(got)
    _lib.call("ht_tomo_RT_coeffx", t._h, _lib.ptr(y), _lib.ptr(scaled), nz, 0.37, st)
    out = torch.empty_like(got)
    _lib.call("ht_shift_coeff_z", sh._hc, _lib.ptr(scaled), _lib.ptr(out), n * n, st)
    assert rel_l2(out.cpu().numpy(), 0.37 * ref.cpu().numpy()) < 1e-5


@pytest.mark.parametrize("tag", ["a", "b"])
def test_rec_tomo_matches_reference(golden, tag):
    """Tomo.rec_tomo (tomo.py:185-210), the CG initial guess, on a noisy phantom
    sinogram, complex and real.  One iteration matches the reference's run to
    1e-5.  CG amplifies the FP32 rounding of the operators and, in the
    reference, of its FP32 inner products (utils.redot through cp.vdot; FP64
    here): after 6 iterations the bound is 1e-4 against the FP64 oracle's CG
    (measured 4-5e-5), as for BH, and 2e-4 against the reference's run
    (measured 8-10e-5)."""
    from holotomocupy_b200 import Tomo
    g = golden("rectomo")
    n, nz, ntheta, niter = [int(v) for v in g[f"{tag}_dims"]]
    t = Tomo(n, nz, g[f"{tag}_theta"], 1)
    d = torch.from_numpy(g[f"{tag}_d"]).cuda()
    assert rel_l2(t.rec_tomo(d, 1).cpu().numpy(), g[f"{tag}_u1"]) < 1e-5
    u = t.rec_tomo(d, niter).cpu().numpy()
    o = O.Tomo(n, nz, g[f"{tag}_theta"], 1, "complex128")
    ref64 = o.rec_tomo(g[f"{tag}_d"].astype("complex128" if tag == "a" else "float64"), niter)
    assert rel_l2(u, ref64) < 1e-4
    assert rel_l2(u, g[f"{tag}_u"]) < 2e-4


def test_R_RT_by_slabs_equal_whole_volume():
    """A Tomo whose workspace holds 8 slices transforms a 20-slice volume slab by
    slab into the same sinogram (and back) as one holding all 20."""
    from holotomocupy_b200 import Tomo
    n, nz, ntheta = 64, 20, 48
    rng = np.random.default_rng(9)
    theta = np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")
    cn = lambda *s: torch.from_numpy((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype("complex64")).cuda()
    x, y = cn(nz, n, n), cn(ntheta, nz, n)
    whole, slabs = Tomo(n, nz, theta, 0.9), Tomo(n, 8, theta, 0.9)
    assert rel_l2(slabs.R(x).cpu().numpy(), whole.R(x).cpu().numpy()) < 1e-7
    assert rel_l2(slabs.RT(y).cpu().numpy(), whole.RT(y).cpu().numpy()) < 1e-7


@pytest.mark.parametrize("n,ntheta,nz", [(18, 20, 1), (24, 5, 4), (32, 100, 5), (48, 33, 8), (64, 150, 9),
                                         (64, 7, 16), (96, 31, 17), (128, 400, 33)])
def test_R_RT_over_slice_batches(n, ntheta, nz):
    """Slice counts around the interleaves of 4, 8 and 16, and angles from dense
    (neighbouring lines share windows; lists near the centre longer than a
    lane group takes) to sparse and unsorted, against the oracle."""
    from holotomocupy_b200 import Tomo
    rng = np.random.default_rng(n + nz)
    theta = np.linspace(0, np.pi, ntheta, endpoint=False)
    if nz % 2:
        theta = rng.permutation(theta + rng.uniform(-0.4, 0.4, ntheta) * np.pi / ntheta) + 2 * np.pi * (nz % 3 - 1)
    theta = theta.astype("float32")
    t = Tomo(n, nz, theta, 1)
    o = O.Tomo(n, nz, theta, 1, "complex64")
    x = (rng.standard_normal((nz, n, n)) + 1j * rng.standard_normal((nz, n, n))).astype("complex64")
    y = (rng.standard_normal((ntheta, nz, n)) + 1j * rng.standard_normal((ntheta, nz, n))).astype("complex64")
    assert rel_l2(t.R(torch.from_numpy(x).cuda()).cpu().numpy(), o.R(x)) < TOL
    assert rel_l2(t.RT(torch.from_numpy(y).cuda()).cpu().numpy(), o.RT(y)) < TOL


@pytest.mark.parametrize("dtype", ["float32", "complex64"])
@pytest.mark.parametrize("kind", ["host", "pinned", "strided", "wider type", "matching"])
def test_R_RT_out_arrays(dtype, kind):
    """out= on the host, strided, of a wider type or matching, by whole volumes
    and by slabs: it holds the result when the call returns, and is returned; a
    matching one is written in place and its version counts up."""
    from holotomocupy_b200 import Tomo
    n, nz, ntheta = 32, 6, 32
    rng = np.random.default_rng(11)
    theta = np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")
    x, y = rng.standard_normal((nz, n, n)), rng.standard_normal((ntheta, nz, n))
    if dtype == "complex64":
        x, y = x + 1j * rng.standard_normal(x.shape), y + 1j * rng.standard_normal(y.shape)
    x, y = (torch.from_numpy(a.astype(dtype)).cuda() for a in (x, y))
    for t in (Tomo(n, nz, theta, 0.9), Tomo(n, 4, theta, 0.9)):
        for op, a in ((t.R, x), (t.RT, y)):
            ref = op(a)
            out = {"host": lambda: torch.empty(ref.shape, dtype=ref.dtype),
                   "pinned": lambda: torch.empty(ref.shape, dtype=ref.dtype, pin_memory=True),
                   "strided": lambda: torch.empty(ref.shape + (2,), dtype=ref.dtype, device="cuda")[..., 1],
                   "wider type": lambda: torch.empty(ref.shape, dtype=torch.promote_types(ref.dtype, torch.float64),
                                                     device="cuda"),
                   "matching": lambda: torch.empty_like(ref)}[kind]()
            version = out._version
            assert op(a, out=out) is out and out._version > version
            assert torch.equal(out.to(ref.device, ref.dtype), ref)


@pytest.mark.parametrize("dtype", ["float32", "complex64"])
@pytest.mark.parametrize("capacity", [10, 24])
def test_R_RT_out_over_the_input(dtype, capacity):
    """out= the input itself, or an array that starts inside it, in one slab and
    in three: the result of a separate out."""
    from holotomocupy_b200 import Tomo
    n = 24   # as many angles and slices as cells: R and R^T keep the shape
    rng = np.random.default_rng(12)
    t = Tomo(n, capacity, np.linspace(0, np.pi, n, endpoint=False).astype("float32"), 0.9)
    x = rng.standard_normal((n, n, n))
    if dtype == "complex64":
        x = x + 1j * rng.standard_normal(x.shape)
    x = torch.from_numpy(x.astype(dtype)).cuda()
    for op in (t.R, t.RT):
        y = x.clone()
        ref = op(x)
        assert torch.equal(op(y, out=y), ref)
        big = torch.cat([x.reshape(-1), x.reshape(-1)[:5]])
        view = big[5:].view(n, n, n)
        assert torch.equal(op(big[:n ** 3].view(n, n, n), out=view), ref)


@pytest.mark.parametrize("dtype", ["float32", "complex64"])
@pytest.mark.parametrize("nz", [17, 20, 21])
def test_R_RT_remainder_run_at_1024(dtype, nz):
    """Up to four slices past a multiple of 16 run by themselves at 1024^2: the
    slices of a call of them alone, in volumes taller than the call too."""
    from holotomocupy_b200 import Tomo
    n, ntheta = 1024, 7
    theta = np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")
    g = torch.Generator(device="cuda").manual_seed(nz)
    dt = getattr(torch, dtype)
    x = torch.randn(nz, n, n, dtype=dt, device="cuda", generator=g)
    y = torch.randn(ntheta, nz, n, dtype=dt, device="cuda", generator=g)
    t, one, part = Tomo(n, nz, theta, 0.9), Tomo(n, 16, theta, 0.9), Tomo(n, 18, theta, 0.9)
    for op, a, ax in (("R", x, 0), ("RT", y, 1)):
        pieces = [getattr(one, op)(a.narrow(ax, z, min(16, nz - z)).contiguous()) for z in (0, 16)]
        ref = torch.cat(pieces, dim=1 - ax)
        for tomo in (t, part):   # 18 slices of capacity: 16 + 2 of the call, then the rest
            got = getattr(tomo, op)(a)
            assert rel_l2(got.cpu().numpy(), ref.cpu().numpy()) < 1e-6
            # the last slice alone: its error is not hidden by the others'
            assert rel_l2(got.select(1 - ax, nz - 1).cpu().numpy(), ref.select(1 - ax, nz - 1).cpu().numpy()) < 1e-6


@pytest.mark.parametrize("n,nz", [(256, 17), (256, 24), (1024, 9), (1024, 20), (1024, 21)])
def test_workspace_slices(n, nz):
    """The memory a Tomo takes beyond one of four slices is that of the slices
    serving counts."""
    from holotomocupy_b200 import Tomo
    from holotomocupy_b200.serving import radon_slices
    theta = np.linspace(0, np.pi, 64, endpoint=False).astype("float32")

    def held(nz):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0] + torch.cuda.memory_reserved()
        t = Tomo(n, nz, theta, 0.9)
        return free - torch.cuda.mem_get_info()[0] - torch.cuda.memory_reserved(), t
    base, _ = held(4)
    got, _ = held(nz)
    want = (radon_slices(n, nz) - 4) * (6 * n + 64) * n * 8
    assert abs(got - base - want) < 0.02 * want + (8 << 20)   # allocations come in 2 MiB pages


@pytest.mark.parametrize("n,nz,less", [(32, 20, 16), (32, 13, 8)])
def test_tomo_without_room_for_the_rounded_workspace(monkeypatch, n, nz, less):
    """Where the workspace of all slices has no room, the whole groups of them run
    slab by slab; another failure, and one of the smallest group, is raised."""
    from holotomocupy_b200 import Tomo, _lib
    theta = np.linspace(0, np.pi, 12, endpoint=False).astype("float32")
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(nz, n, n, dtype=torch.complex64, device="cuda", generator=g)
    ref = Tomo(n, nz, theta, 0.9).R(x)
    call = _lib.call

    def failing(limit, message):
        def f(name, *args):
            if name == "ht_tomo_create" and args[1] > limit:
                raise _lib.HoloError(f"{name} failed with status 2: {message}")
            return call(name, *args)
        return f
    monkeypatch.setattr(_lib, "call", failing(less, "ht_tomo_create: out of memory"))
    t = Tomo(n, nz, theta, 0.9)
    assert t._nz == less
    assert rel_l2(t.R(x).cpu().numpy(), ref.cpu().numpy()) < 1e-6
    for limit, message in ((less - 1, "out of memory"), (less, "unknown error")):
        monkeypatch.setattr(_lib, "call", failing(limit, message))
        with pytest.raises(_lib.HoloError, match=message):
            Tomo(n, nz, theta, 0.9)


@pytest.mark.parametrize("n,ntheta", [(64, 300), (64, 90), (128, 401)])
def test_R_RT_over_a_full_turn(n, ntheta):
    """Angles over 2 pi, sorted and not: theta and theta + pi share a line from
    opposite ends."""
    from holotomocupy_b200 import Tomo
    rng = np.random.default_rng(ntheta)
    theta = np.linspace(0, 2 * np.pi, ntheta, endpoint=False)
    theta = (rng.permutation(theta) if ntheta % 2 else theta).astype("float32")
    nz = 9
    t, o = Tomo(n, nz, theta, 1), O.Tomo(n, nz, theta, 1, "complex64")
    x = (rng.standard_normal((nz, n, n)) + 1j * rng.standard_normal((nz, n, n))).astype("complex64")
    y = (rng.standard_normal((ntheta, nz, n)) + 1j * rng.standard_normal((ntheta, nz, n))).astype("complex64")
    assert rel_l2(t.R(torch.from_numpy(x).cuda()).cpu().numpy(), o.R(x)) < TOL
    assert rel_l2(t.RT(torch.from_numpy(y).cuda()).cpu().numpy(), o.RT(y)) < TOL


@pytest.mark.parametrize("dtype", ["float32", "complex64"])
@pytest.mark.parametrize("n,ntheta,nz,slab", [(32, 100, 5, 4), (48, 33, 8, 8), (64, 150, 9, 4), (96, 31, 17, 16),
                                              (64, 48, 20, 8)])
def test_R_RT_fbp_over_types_and_slabs(dtype, n, ntheta, nz, slab):
    """Real and complex volumes, whole and by slabs, at slice counts around the
    interleaves: R, R^T and filtered back-projection against the FP64 oracle,
    a real volume's as the real part of a complex one's."""
    from holotomocupy_b200 import Tomo
    rng = np.random.default_rng(n + nz)
    theta = np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")
    x, y = rng.standard_normal((nz, n, n)), rng.standard_normal((ntheta, nz, n))
    if dtype == "complex64":
        x, y = x + 1j * rng.standard_normal(x.shape), y + 1j * rng.standard_normal(y.shape)
    x, y = x.astype(dtype), y.astype(dtype)
    wide = np.complex128 if dtype == "complex64" else np.float64
    o = O.Tomo(n, nz, theta, 0.9, "complex128")
    refs = [o.R(x.astype(wide)), o.RT(y.astype(wide))]
    refs += [o.fbp(y.astype(wide), f) for f in ("ramp", "shepp", "parzen")]
    for t in (Tomo(n, nz, theta, 0.9), Tomo(n, slab, theta, 0.9)):
        xt, yt = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        got = [t.R(xt), t.RT(yt)] + [t.fbp(yt, f) for f in ("ramp", "shepp", "parzen")]
        for a, b in zip(got, refs):
            assert a.dtype == xt.dtype and rel_l2(a.cpu().numpy(), b) < TOL
        if dtype == "float32":
            assert rel_l2(t.R(xt.to(torch.complex64)).real.cpu().numpy(), got[0].cpu().numpy()) < 1e-7
            assert rel_l2(t.RT(yt.to(torch.complex64)).real.cpu().numpy(), got[1].cpu().numpy()) < 1e-7


@pytest.mark.parametrize("dtype", ["float32", "complex64"])
@pytest.mark.parametrize("n", [18, 96, 512])
def test_filter_sino_matches_oracle(dtype, n):
    """The detector filter alone (ht_filter_rows)."""
    from holotomocupy_b200 import Tomo
    theta = np.linspace(0, np.pi, 5, endpoint=False).astype("float32")
    rng = np.random.default_rng(n)
    d = rng.standard_normal((5, 3, n))
    d = (d + 1j * rng.standard_normal(d.shape) if dtype == "complex64" else d).astype(dtype)
    t, o = Tomo(n, 3, theta, 1), O.Tomo(n, 3, theta, 1, "complex128")
    for f in ("ramp", "shepp", "parzen"):
        got = t._filter_sino(torch.from_numpy(d).cuda(), f)
        assert rel_l2(got.cpu().numpy(), o.filter_sino(d.astype(np.complex128 if dtype == "complex64" else float), f)) < 1e-6
