"""The blocked kernels of the differentiable path at the sizes where they can go wrong, against
float64 references: the Gaussian blur and its adjoint (line lengths around the group and tile
sizes, the smallest radius of the blocked kernel and one below it), the soft-argmax (few cells,
values that leave the float range between), and the NLPAR average, adjoint and weight gradient
(the smallest grids of each radius, ragged pattern sizes).

Bars are forward error bounds of the float sums: (terms + roundings of a term) x 2^-24 times the
sum of the terms' magnitudes, with the exponential's own error (2 ulp) and its rounded argument
for the soft-argmax."""
import numpy as np
import pytest

from pyebsdindex_gb300 import diff

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


def _blur_matrix(taps, L):
    r = len(taps) // 2
    A, B = np.zeros((L, L)), np.zeros((L, L))
    for o in range(L):
        for t in range(-r, r + 1):
            q = abs(o + t)
            q = 2 * (L - 1) - q if q >= L else q
            A[o, q] += float(taps[t + r])
            B[o, q] += abs(float(taps[t + r]))
    return A, B


@pytest.mark.parametrize("n,h,w,r", [(1, 4, 5, 3), (3, 7, 9, 3), (2, 8, 16, 7), (5, 61, 60, 15), (1, 33, 31, 30),
                                     (33, 40, 64, 16), (2, 17, 200, 5), (4, 12, 13, 2), (1, 800, 6, 4)])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("adjoint", [False, True])
def test_blur(cuda, n, h, w, r, axis, adjoint):
    import torch
    L = h if axis == 0 else w
    r = min(r, L - 1)
    g = np.random.default_rng(n * 1000 + h + w)
    taps = g.normal(size=2 * r + 1).astype(np.float32)
    x = g.normal(size=(n, h, w)).astype(np.float32)
    y = diff._blur(diff._bind(), torch.from_numpy(x.reshape(n, -1)).to(cuda), torch.from_numpy(taps).to(cuda), r, h, w,
                   axis, adjoint).cpu().numpy().reshape(n, h, w)
    A, B = _blur_matrix(taps, L)
    if adjoint:
        A, B = A.T, B.T
    eq = "oq,nqx->nox" if axis == 0 else "oq,nyq->nyo"
    want, mag = np.einsum(eq, A, x.astype(np.float64)), np.einsum(eq, B, np.abs(x).astype(np.float64))
    assert np.all(np.abs(y - want) <= (4 * r + 4) * U * mag)


@pytest.mark.parametrize("adjoint", [False, True])
def test_blur_keeps_nonfinite_local(cuda, adjoint):
    """A value that is not finite reaches the outputs within r of it and no other."""
    import torch
    n, h, w, r = 2, 40, 50, 5
    x = np.ones((n, h, w), np.float32)
    x[1, 20, 30] = np.inf
    taps = torch.full((2 * r + 1,), 0.1, device=cuda)
    for axis in (0, 1):
        y = diff._blur(diff._bind(), torch.from_numpy(x.reshape(n, -1)).to(cuda), taps, r, h, w, axis, adjoint)
        bad = ~np.isfinite(y.cpu().numpy().reshape(n, h, w))
        want = np.zeros_like(bad)
        if axis == 0:
            want[1, 15:26, 30] = True
        else:
            want[1, 20, 25:36] = True
        assert np.array_equal(bad, want)


@pytest.mark.parametrize("n,ncell,keep,tau,scale", [(1, 1, 1, 1.0, 1.0), (3, 31, 31, 0.3, 5.0), (2, 257, 200, 2.0, 50.0),
                                                    (5, 1000, 700, 50.0, 30.0), (4, 3000, 2999, 1e-3, 1.0),
                                                    (2, 300, 299, 1.0, 1e32)])
def test_softargmax(cuda, n, ncell, keep, tau, scale):
    import torch
    from pyebsdindex_gb300 import _lib
    g = np.random.default_rng(ncell)
    c = (g.normal(size=(n, ncell)) * scale).astype(np.float32)
    cells = np.sort(g.permutation(ncell)[:keep]).astype(np.int32)
    ct, ci = torch.from_numpy(c).to(cuda), torch.from_numpy(cells).to(cuda)
    J = torch.empty(n, dtype=torch.float64, device=cuda)
    grad = torch.zeros_like(ct)
    _lib.check(diff._bind().ebsd_softargmax(0, ct.data_ptr(), n, ncell, ci.data_ptr(), keep, tau, J.data_ptr(),
                                            grad.data_ptr(), torch.cuda.current_stream().cuda_stream), "softargmax")
    v = c[:, cells].astype(np.float64)
    a = (v - v.max(1, keepdims=True)) / tau
    e = np.exp(a)
    S = e.sum(1, keepdims=True)
    s = e / S
    want = (s * v).sum(1, keepdims=True)
    de = (np.abs(a) * U * 1.01 + 4 * U) * e + 1e-44
    dJ = 1.05 * (de * np.abs(v - want)).sum(1, keepdims=True) / S + 1e-12 * np.abs(v).max(1, keepdims=True)
    assert np.all(np.abs(J.cpu().numpy() - want[:, 0]) <= dJ[:, 0])
    f = 1.0 + (v - want) / tau
    rs = de / S + s * de.sum(1, keepdims=True) / S
    tol = 1.05 * (rs * np.abs(f) + s * dJ / tau) + 2 * U * np.abs(s * f) + 1e-44
    got = grad.cpu().numpy()
    assert np.all(np.abs(got[:, cells] - s * f) <= tol)
    off = np.ones(ncell, bool)
    off[cells] = False
    assert np.all(got[:, off] == 0)


def _window(i, sr, n):
    a = min(max(i - sr, 0), n - (2 * sr + 1))
    return a, a + 2 * sr + 1


def _slots(nr, nc, sr):
    out = np.zeros((nr * nc, (2 * sr + 1) ** 2), np.int64)
    for p in range(nr * nc):
        ys, ye = _window(p // nc, sr, nr)
        xs, xe = _window(p % nc, sr, nc)
        out[p] = [j * nc + i for j in range(ys, ye) for i in range(xs, xe)]
    return out


GRIDS = [(3, 3, 5, 1), (4, 7, 1025, 1), (5, 5, 64, 2), (6, 9, 1300, 2), (7, 8, 77, 3), (9, 11, 2052, 4), (3, 2, 33, 0)]


@pytest.mark.parametrize("nr,nc,npx,sr", GRIDS)
def test_average_and_adjoint(cuda, nr, nc, npx, sr):
    import torch
    from pyebsdindex_gb300 import _lib
    lib, g = diff._bind(), np.random.default_rng(npx)
    x = g.normal(size=(nr * nc, npx)).astype(np.float32)
    slots = _slots(nr, nc, sr)
    w = g.random(slots.shape).astype(np.float32)
    A = np.zeros((nr * nc, nr * nc))
    for p in range(nr * nc):
        A[p, slots[p]] = w[p]
    xt, wt = torch.from_numpy(x).to(cuda), torch.from_numpy(w).to(cuda)
    st = torch.cuda.current_stream().cuda_stream
    for fn, M in ((lib.ebsd_nlpar_apply, A), (lib.ebsd_nlpar_apply_t, A.T)):
        y = torch.empty_like(xt)
        _lib.check(fn(xt.data_ptr(), nr, nc, npx, wt.data_ptr(), sr, y.data_ptr(), st), "apply")
        terms = int((M != 0).sum(1).max())
        assert np.all(np.abs(y.cpu().numpy() - M @ x.astype(np.float64)) <= (2 * terms + 2) * U * (M @ np.abs(x)))


@pytest.mark.parametrize("nr,nc,npx,sr", GRIDS)
@pytest.mark.parametrize("f64", [False, True])
def test_weights_grad(cuda, nr, nc, npx, sr, f64):
    import torch
    from pyebsdindex_gb300 import _lib
    rng, n, dt = np.random.default_rng(npx + sr), nr * nc, np.float64 if f64 else np.float32
    lam, datamax, sat = 0.9, 200.0, 1
    g, x = rng.normal(size=(n, npx)).astype(dt), rng.integers(0, 201, size=(n, npx)).astype(dt)
    slots = _slots(nr, nc, sr)
    ws = slots.shape[1]
    w, m, dS, dg = (rng.random((n, ws)).astype(np.float32) for _ in range(4))
    centre = slots == np.arange(n)[:, None]
    dS[centre] = dg[centre] = 0
    arg = np.full(n, -1, np.int32)
    for p in range(n):
        near = [j * nc + i for j in range(max(p // nc - 1, 0), min(p // nc + 2, nr))
                for i in range(max(p % nc - 1, 0), min(p % nc + 2, nc)) if j * nc + i != p]
        if p % 5:
            arg[p] = near[int(rng.integers(len(near)))]
    nsig = rng.integers(1, npx + 1, size=n).astype(np.float32)
    mask = (rng.random(npx) < 0.8).astype(np.uint8)
    dev = [torch.from_numpy(a).to(cuda) for a in (g, x, w, m, dS, dg, mask, arg, nsig)]
    scr = torch.empty(3 * n * ws + n, dtype=torch.float64, device=cuda)
    gl, gx = torch.empty(n, dtype=torch.float64, device=cuda), torch.empty_like(dev[0])
    _lib.check(diff._bind().ebsd_nlpar_weights_grad(
        int(f64), dev[0].data_ptr(), dev[1].data_ptr(), nr, nc, npx, sr, *(t.data_ptr() for t in dev[2:6]), lam,
        dev[6].data_ptr(), datamax, sat, dev[7].data_ptr(), dev[8].data_ptr(), scr.data_ptr(), gl.data_ptr(),
        gx.data_ptr(), torch.cuda.current_stream().cuda_stream), "weights_grad")
    u = 2.0 ** -53 * 8 if f64 else U
    g, x, w, m, dS, dg = (a.astype(np.float64) for a in (g, x, w, m, dS, dg))
    G = np.einsum("pk,pck->pc", g, x[slots])
    eG = (2 if not f64 else npx) * u * np.einsum("pk,pck->pc", np.abs(g), np.abs(x[slots]))
    dev_, eD = G - (w * G).sum(1, keepdims=True), eG + (w * eG).sum(1, keepdims=True)
    glam = (w * 2 / lam ** 3 * m * dev_).sum(1)
    assert np.all(np.abs(gl.cpu().numpy() - glam) <= 1.01 * (w * 2 / lam ** 3 * m * eD).sum(1) + 1e-9 * np.abs(glam) + 1e-9)
    al, be = -w / lam ** 2 * dev_ * dS, -w / lam ** 2 * dev_ * dg
    eal, ebe = w / lam ** 2 * eD * dS, w / lam ** 2 * eD * dg
    gam, egam = be.sum(1), ebe.sum(1)
    for p in range(n):
        for c in range(ws):
            if slots[p, c] != p:
                gam[slots[p, c]] += be[p, c]
                egam[slots[p, c]] += ebe[p, c]
    mxw, mxs = float(np.float32(datamax) * np.float32(0.999)), float(np.float32(datamax) * np.float32(0.9961))
    want, tol, terms = np.zeros((n, npx)), np.zeros((n, npx)), np.zeros(n)

    def pair(q, o, c, ec, lim):
        ok = (mask != 0) & (x[q] < lim) & (x[o] < lim)
        want[q] += c * (x[q] - x[o]) * ok
        tol[q] += (ec + abs(c) * 4 * u) * np.abs(x[q] - x[o]) * ok
        mag[q] += abs(c) * np.abs(x[q] - x[o]) * ok
        terms[q] += 1

    mag = np.zeros((n, npx))
    for p in range(n):
        for c in range(ws):
            o = slots[p, c]
            if o != p:
                pair(p, o, 2 * al[p, c], 2 * eal[p, c], mxw)
                pair(o, p, 2 * al[p, c], 2 * eal[p, c], mxw)
        if arg[p] >= 0:
            pair(p, arg[p], gam[p] / nsig[p], egam[p] / nsig[p], mxs)
            pair(arg[p], p, gam[p] / nsig[p], egam[p] / nsig[p], mxs)
    tol += (terms[:, None] + 1) * u * mag
    assert np.all(np.abs(gx.cpu().numpy() - want) <= 1.01 * tol + 1e-12 * mag)


@pytest.mark.parametrize("nr,nc,npx,nind,sr", [(3, 3, 5, 5, 1), (4, 7, 1025, 900, 1), (5, 5, 64, 33, 2), (6, 70, 130, 65, 2),
                                               (7, 8, 77, 31, 3), (9, 61, 300, 96, 3), (35, 7, 40, 1, 3), (5, 6, 9, 0, 2)])
@pytest.mark.parametrize("given", [False, True])
def test_sigma_weights_equal_the_pairwise_kernels(cuda, nr, nc, npx, nind, sr, given):
    """Bit for bit, with saturated values and a NaN among the patterns."""
    import torch
    from pyebsdindex_gb300 import _lib
    lib, g, n, ws = diff._bind(), np.random.default_rng(npx), nr * nc, (2 * sr + 1) ** 2
    x = g.integers(0, 201, size=(n, npx)).astype(np.float32)
    x[n // 2, npx // 2] = np.nan
    xt = torch.from_numpy(x).to(cuda)
    ind = torch.from_numpy(np.sort(g.permutation(npx)[:nind]).astype(np.int32)).to(cuda)
    ip = (ind if nind else torch.zeros(1, dtype=torch.int32, device=cuda)).data_ptr()
    st = torch.cuda.current_stream().cuda_stream

    def outs():
        sig2 = torch.full((n,), 3.0, device=cuda)
        return [sig2, torch.zeros(n, dtype=torch.int32, device=cuda), torch.zeros(n, device=cuda)] + [
            torch.zeros((n, ws), device=cuda) for _ in range(4)]
    a, b = outs(), outs()
    if not given:
        _lib.check(lib.ebsd_nlpar_sigma_arg(xt.data_ptr(), nr, nc, npx, ip, nind, 200.0, 1,
                                            *(t.data_ptr() for t in a[:3]), st), "sigma_arg")
    _lib.check(lib.ebsd_nlpar_weights_d(xt.data_ptr(), nr, nc, npx, ip, nind, 200.0, 0.9, sr, 0.1, a[0].data_ptr(), 1,
                                        *(t.data_ptr() for t in a[3:]), st), "weights_d")
    work = torch.empty(int(lib.ebsd_nlpar_sigma_weights_d_work(nr, nc, sr)), device=cuda)
    _lib.check(lib.ebsd_nlpar_sigma_weights_d(xt.data_ptr(), nr, nc, npx, ip, nind, 200.0, 0.9, sr, 0.1, int(not given),
                                              1, work.data_ptr(), *(t.data_ptr() for t in b), st), "sigma_weights_d")
    for s, t in zip(a, b):
        assert torch.equal(s.view(torch.int32), t.view(torch.int32))


@pytest.mark.parametrize("nrows,ncols,width", [(1, 1, 0), (1, 7, 1), (37, 50, 0), (61 * 9, 300, 61), (64, 20, 8), (35, 64, 5),
                                               (33, 12, 33)])
@pytest.mark.parametrize("f64", [False, True])
def test_linop_tiles_equal_rows(cuda, nrows, ncols, width, f64):
    """Tiles of neighbouring rows, ragged row lengths and empty rows: the same bits as a thread a row."""
    import torch
    g = np.random.default_rng(nrows)
    cnt = g.integers(0, min(ncols, 40) + 1, size=nrows)
    cnt[nrows // 2] = 0
    rowptr = np.concatenate([[0], np.cumsum(cnt)])
    col = np.concatenate([np.sort(g.permutation(ncols)[:c]) for c in cnt] + [[]]).astype(np.int32)
    op = diff.LinOp(rowptr, col, g.normal(size=len(col)).astype(np.float32), (nrows, ncols), width=width)
    for n in (1, 31, 33, 64, 65, 127, 130, 257):
        x = torch.from_numpy(g.normal(size=(n, ncols))).to(cuda, torch.float64 if f64 else torch.float32)
        assert torch.equal(op(x), op.apply_rows(x)), n
