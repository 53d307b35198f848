"""te_w_solve_static_scratch against the same solve in binary64, at the edges of its two forms:
tiles of 32 columns in shared memory up to nz = 200, the scratch array above."""
import ctypes

import numpy as np
import pytest

SCALE = {'pk1': 2.5e-3, 'pk2': -2.5e-3, 'qk': 2.5e-4, 'mm': 500.0, 'fpk': 1e-5, 'wten': 1e-2, 'pp3d': 1e-4, 'w': 1.0}


# one tile with one column; more tiles than resident blocks, the last one ragged; columns that
# fill the two buffers, and one level more; fewer levels than loader warps; nz = 3
@pytest.mark.gpu
@pytest.mark.parametrize('nx,ny,nz', [(1, 1, 5), (203, 190, 9), (40, 24, 200), (24, 20, 201), (31, 33, 6), (65, 3, 3),
                                      (32, 8, 80)])
def test_solve_against_binary64(nx, ny, nz):
    import torch
    from thunderengine_web_b200.replayer import TeWSolveFields, load_library
    rng = np.random.default_rng(nx * 1000 + nz)
    f = {}
    for n, s in SCALE.items():
        x = rng.random((nz + 1, ny + 7, nx + 7))
        f[n] = ((x + 0.5 if n in ('pk1', 'pk2', 'mm') else x - 0.5) * s).astype(np.float32)
    dev = {n: torch.from_numpy(x).cuda() for n, x in f.items()}
    args = TeWSolveFields(*[dev[n].data_ptr() for n in ('pk1', 'pk2', 'qk', 'mm', 'fpk', 'wten', 'pp3d', 'w')])
    dts, alph, beta = (np.float64(np.float32(x)) for x in (0.375, 0.6, 0.4))
    err = ctypes.create_string_buffer(256)
    rc = load_library().te_w_solve_static_scratch(ctypes.byref(args), nx, ny, nz, dts, alph, beta, None, err, 256)
    assert rc == 0, err.value.decode()
    torch.cuda.synchronize()
    got = dev['w'].cpu().numpy()
    box = (slice(None), slice(3, 3 + ny), slice(3, 3 + nx))
    pk1, pk2, qk, mm, fpk, wten, pp, w0 = (f[n][box].astype(np.float64)
                                           for n in ('pk1', 'pk2', 'qk', 'mm', 'fpk', 'wten', 'pp3d', 'w'))
    a, d, s, asq = pk1 + qk, pk2 - qk, pp + fpk, alph * alph
    want = f['w'].astype(np.float64)
    ca, cb = np.zeros_like(a), np.zeros_like(a)
    for k in range(1, nz):
        aa, cc, bb = -asq * mm[k] * a[k - 1], asq * mm[k] * d[k], 1.0 - asq * mm[k] * (d[k - 1] - a[k])
        dd = w0[k] + dts * wten[k] - beta * mm[k] * (pp[k] - pp[k - 1]) - alph * mm[k] * (s[k] - s[k - 1])
        den = bb + aa * ca[k - 1]
        ca[k], cb[k] = -cc / den, (dd - aa * cb[k - 1]) / den
    x = np.zeros_like(a[0])
    want[0][box[1:]] = want[nz][box[1:]] = 0.0
    for k in range(nz - 1, 0, -1):
        x = cb[k] + (ca[k] * x if k < nz - 1 else 0.0)
        want[k][box[1:]] = x
    # a few roundings per level, carried down the column: nz * 2^-23 of the largest w
    assert np.abs(got - want).max() <= nz * 2.0 ** -23 * np.abs(want).max()
    outside = np.ones(want.shape, bool)
    outside[box] = False
    assert np.array_equal(got[outside], f['w'][outside])   # halos untouched
