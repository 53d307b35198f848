"""Performance cases: what a user of this library has it do, through its public calls.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare``
makes what a program has in hand before the call (planned players whose state is on the
GPU), ``run`` is one pass, ``work`` the bytes and operations a pass cannot do without and
``exact`` the 64-bit result where plain torch gives it.

Kinds of cases:

* ``step``: one large step of a synthetic storm (``Replayer.encode_steps``), the library's
  main path: exact or fused mode, moist or dry, packed or aligned rows, from the smallest
  grid the tests use to the large domain;
* ``physics``: a recorded full-physics step (open or mixed boundaries, turbulence,
  microphysics), optionally with the display diagnostic (``Replayer.encode_diag``);
* ``adjoint``: a window of dynamics-core steps and its gradient
  (``Replayer.adjoint_forward`` / ``adjoint_backward``);
* ``ensemble``: members of different sizes advanced together (``Ensemble.run``);
* ``wsolve``: the implicit column solve on fields of the caller's own
  (``te_w_solve_static_scratch``).
"""
import ctypes
import functools
import gzip
import json
import math
import os
import random

import numpy as np
import torch

from thunderengine_web_b200 import scenario, timestep
from thunderengine_web_b200.replayer import (TE_MODE_EXACT, TE_MODE_FUSED, Ensemble, Replayer, TeWSolveFields,
                                             load_library)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RECORDINGS = os.path.join(ROOT, 'tests', 'golden')
MODES = {'exact': TE_MODE_EXACT, 'fused': TE_MODE_FUSED}
# prognostic and thermodynamic fields a program reads after a step
MOIST_OUT = ('th', 'qv', 'u', 'v', 'w', 'pp3d', 'prs', 'rho')
DRY_OUT = ('th', 'u', 'v', 'w', 'pp3d', 'prs', 'rho')
PHYSICS_OUT = ('th', 'qv', 'qc', 'qr', 'qi', 'qs', 'qg', 'nci', 'ncs', 'ncr', 'ncg', 'tke', 'u', 'v', 'w', 'pp3d',
               'prs', 'rho')
WSOLVE_IN = ('pk1', 'pk2', 'qk', 'mm', 'fpk', 'wten', 'pp3d')
WSOLVE_MOST = 8388608   # nx * ny * (nz - 2) the static scratch holds


def _step(name, nx, ny, nz, mode, dx=500.0, dz=250.0, dt=3.0, nsound=8, us=25.0, dry=False, align=False):
    c = dict(kind='step', nx=nx, ny=ny, nz=nz, mode=mode, dx=dx, dz=dz, dt=dt, nsound=nsound, us=us, dry=dry, align=align)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest grid of the tests: a step is launch latency only
        _step('tiny-exact', 12, 10, 8, 'exact', dx=1000.0, dz=500.0, dt=6.0, nsound=6, us=20.0),
        # odd sizes: no extent is a multiple of a warp, a tile or a pass of levels
        _step('odd-fused', 37, 29, 13, 'fused'),
        # the small configuration (scenario.SMALL): a quick run on a coarse grid
        _step('small-fused', 64, 64, 40, 'fused', dx=1000.0, dz=500.0, dt=6.0, nsound=6, us=20.0),
        # the mode a player has without set_mode, on an ordinary grid: every dispatch of the tape
        _step('ordinary-exact', 128, 128, 64, 'exact'),
        # the dry step on the aligned-row layout, ragged extents
        _step('dry-aligned-fused', 150, 101, 48, 'fused', dry=True, align=True),
        # the benchmark's configuration (scenario.AT_SCALE)
        _step('at-scale-fused', 256, 256, 80, 'fused'),
        # the large domain (scenario.LARGE): 21 GB of state, offsets past 2^32 words
        _step('large-fused', 1024, 1024, 100, 'fused', dx=250.0, dz=200.0, dt=1.5),
        # a recorded full-physics step, open on all sides, as the recording plays it
        dict(name='physics-exact', kind='physics', recording='single_cell', mode='exact', steps=1, diag=False),
        # a frame of the display: a full-physics step periodic in y, then its reflectivity
        dict(name='physics-frame-fused', kind='physics', recording='squall_line', mode='fused', steps=1, diag=True),
        # gradient of a window on the adjoint configuration's grid, two checkpoint blocks
        dict(name='adjoint-window', kind='adjoint', nx=128, ny=128, nz=64, steps=10, every=5),
        # an ensemble of uneven members, one large step of each
        dict(name='ensemble', kind='ensemble', members=12, sizes=7),
        # the column solve on caller-owned fields at the benchmark's size
        dict(name='column-solve', kind='wsolve', nx=256, ny=256, nz=80),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: mostly single steps, sizes spread over the logarithm of their range."""
    p = rng.random()
    if p < 0.6:
        nz = _log(rng, 8, 100)
        fine = rng.random() < 0.5
        return _step(None, _log(rng, 12, 1024), _log(rng, 12, 1024), nz, 'fused' if rng.random() < 0.65 else 'exact',
                     dx=500.0 if fine else 1000.0, dz=min(500.0, (12000.0 if fine else 16000.0) / nz),
                     dt=3.0 if fine else 6.0, nsound=rng.randint(6, 8), us=float(rng.randint(10, 30)),
                     dry=rng.random() < 0.2, align=rng.random() < 0.25)
    if p < 0.74:
        return dict(kind='physics', recording=rng.choice(['single_cell', 'squall_line', 'supercell_stretched']),
                    mode=rng.choice(['exact', 'fused']), steps=rng.randint(1, 4), diag=rng.random() < 0.5)
    if p < 0.84:
        return dict(kind='adjoint', nx=_log(rng, 16, 128), ny=_log(rng, 16, 128), nz=rng.randint(12, 64),
                    steps=rng.randint(2, 10), every=rng.randint(1, 5))
    if p < 0.93:
        return dict(kind='ensemble', members=rng.randint(3, 24), sizes=rng.randrange(1 << 20))
    nz = rng.randint(8, 100)
    nx = _log(rng, 16, 512)
    return dict(kind='wsolve', nx=nx, ny=_log(rng, 12, min(512, WSOLVE_MOST // (nx * (nz - 2)))), nz=nz)


# ------------------------------------------------------------------ inputs


class _Words:
    """Device words of a player as torch sees them, without a copy; they keep the player."""

    def __init__(self, owner, ptr, words):
        self.owner = owner
        self.__cuda_array_interface__ = {'shape': (int(words),), 'typestr': '<f4', 'data': (int(ptr), False), 'version': 3}


def _device_words(r, off, words):
    return torch.as_tensor(_Words(r, r.device_ptr(off), words), device='cuda')


def _field(r, run, name):
    g = run.grid
    off = r.base[run.rec.ids['arena']] + run.fields[name] // 4
    return _device_words(r, off, g.count).view(g.nz + 1, g.strideK, g.strideJ)


@functools.lru_cache(maxsize=64)
def _run(nx, ny, nz, dx, dz, dt, nsound, us, dry=False, align=False, core=False):
    """The encoder's run and its tape as a program keeps them for a configuration."""
    cfg = scenario.Config('case-%dx%dx%d' % (nx, ny, nz), nx, ny, nz, dx, dz, dt, nsound, us, 1, align_rows=align)
    run = timestep.Run(cfg, core=core, moist=not dry)
    return run, json.dumps(run.tape(1))


def _periodic(a, nx, ny):
    h = scenario.HALO
    a[:, :, :h] = a[:, :, nx:nx + h]
    a[:, :, nx + h:nx + 2 * h + 1] = a[:, :, h:2 * h + 1]
    a[:, :h] = a[:, ny:ny + h]
    a[:, ny + h:ny + 2 * h + 1] = a[:, h:2 * h + 1]


def _fill_state(r, run, seed):
    """The storm's start on the device: sounding, sheared wind, warm bubble and +-0.1 K noise
    (scenario.fill_arena with the noise of a torch generator)."""
    g, prof, cfg = run.grid, run.prof, run.cfg
    nx, ny, nz, h = g.nx, g.ny, g.nz, scenario.HALO
    dev = torch.device('cuda')
    for i, name in enumerate(run.rec.buffers):
        if name != 'arena':
            r.upload(i, run.buffer_bytes(name))

    def column(v):
        return torch.from_numpy(np.ascontiguousarray(v, dtype=np.float32)).to(dev)[:, None, None]
    W = nx + 1 + 2 * h
    xh = torch.from_numpy(g.axis(nx, g.dx)[1][h:h + nx]).to(dev).float()
    yh = torch.from_numpy(g.axis(ny, g.dy)[1][h:h + ny]).to(dev).float()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    th = torch.rand((nz, ny, nx), generator=gen, device=dev)
    th.mul_(2.0 * cfg.noise).sub_(cfg.noise)
    for k in range(nz):   # the bubble reaches to 2.8 km
        bz = (float(prof['vg'].zh[k]) - 1400.0) / 1400.0
        if abs(bz) < 1.0:
            beta = torch.sqrt((xh / 10000.0)[None, :] ** 2 + (yh / 10000.0)[:, None] ** 2 + bz * bz)
            th[k] += torch.where(beta < 1.0, cfg.amplitude * torch.cos(0.5 * math.pi * beta) ** 2, 0.0)
    f = _field(r, run, 'th')
    f[:nz, h:h + ny, h:h + nx] = th
    del th
    _periodic(f[:nz, :, :W], nx, ny)
    _field(r, run, 'th_a').copy_(f)
    for names, prof_name in ((('qv', 'qv_a'), 'qv0'), (('u', 'u_a'), 'u0')):
        for n in names:
            if n in run.fields:
                _field(r, run, n)[:nz, :, :W] = column(prof[prof_name])
    p = np.array([scenario.f(scenario.f(scenario.P00) * np.power(x, scenario.f(scenario.CP / scenario.RD)))
                  for x in prof['pi0']], np.float32)
    _field(r, run, 'prs')[:nz, :, :W] = column(p)
    rho = _field(r, run, 'rho')
    rmix = scenario.RD + np.maximum(0.0, prof['qv0']) * scenario.RV
    rho[:nz, :, :W] = column(p) / ((column(prof['th0']) + f[:nz, :, :W]) * column(prof['pi0'] * rmix))
    torch.cuda.synchronize()


@functools.lru_cache(maxsize=None)
def _stream():
    """The program's stream: its players' steps run one after another."""
    return torch.cuda.Stream()


def _player(run, tape, seed, mode):
    r = Replayer(tape)
    r.plan(False)
    r.build()
    _fill_state(r, run, seed)
    r.set_stream(_stream().cuda_stream)
    r.set_mode(MODES[mode])
    return r


def _outputs(r, run, names):
    return {n: _field(r, run, n) for n in names}


@functools.lru_cache(maxsize=None)
def _recording(name):
    d = os.path.join(RECORDINGS, name)
    with open(os.path.join(d, 'tape.json')) as fh:
        text = fh.read()
    with open(os.path.join(RECORDINGS, 'kernels.json')) as fh:
        kernels = fh.read()   # the recordings' kernel table: parameters and per-thread scratch
    tape = json.loads(text)
    state = {}
    for b in tape['buffers']:
        p = os.path.join(d, 'state', '%d.bin.gz' % b['id'])
        if os.path.exists(p):
            with gzip.open(p, 'rb') as fh:
                state[b['id']] = fh.read()
    return tape, text, kernels, state


def _prepare_step(c, seed):
    run, tape = _run(c['nx'], c['ny'], c['nz'], c['dx'], c['dz'], c['dt'], c['nsound'], c['us'], c['dry'], c['align'])
    r = _player(run, tape, seed, c['mode'])
    return {'kind': 'step', 'r': r, 'out': _outputs(r, run, DRY_OUT if c['dry'] else MOIST_OUT)}


def _prepare_physics(c, seed):
    tape, text, kernels, state = _recording(c['recording'])
    r = Replayer(text, kernels)
    r.plan(False)
    r.build()
    for i, b in state.items():
        r.upload(i, b)
    aid = next(b['id'] for b in tape['buffers'] if b['arena'])
    nx, ny, nz = tape['nx'], tape['ny'], tape['nz']
    shape = (nz + 1, ny + 7, nx + 7)

    def field(name):
        return _device_words(r, r.base[aid] + tape['fields'][name] // 4, math.prod(shape)).view(shape)
    gen = torch.Generator(device='cuda')
    gen.manual_seed(int(seed))
    noise = (torch.rand((nz, ny, nx), generator=gen, device='cuda') - 0.5) * 0.2
    for n in ('th', 'th_a'):   # +-0.1 K on the recorded state
        field(n)[:nz, 3:3 + ny, 3:3 + nx] += noise
    torch.cuda.synchronize()
    r.set_stream(_stream().cuda_stream)
    r.set_mode(MODES[c['mode']])
    out = {n: field(n) for n in PHYSICS_OUT + (('dbz',) if c['diag'] else ())}
    return {'kind': 'physics', 'r': r, 'steps': c['steps'], 'diag': c['diag'], 'out': out}


def _prepare_adjoint(c, seed):
    run, tape = _run(c['nx'], c['ny'], c['nz'], 500.0, min(250.0, 16000.0 / c['nz']), 3.0, 8, 25.0, core=True)
    first = _player(run, tape, seed, 'fused')   # the window starts after a regular step
    first.encode_steps(1)
    first.sync()
    r = Replayer(run.tape(1, core=True))
    r.plan(False)
    r.build()
    for i, name in enumerate(run.rec.buffers):
        words = run.buffer_length(name) // 4
        _device_words(r, r.base[i], words).copy_(_device_words(first, first.base[i], words))
    torch.cuda.synchronize()
    r.set_stream(_stream().cuda_stream)   # the mode stays the one adjoint.CoreWindow has
    r.adjoint_forward(1, c['every'])   # lays out the adjoint memory
    r.adjoint_zero()
    r.adjoint_backward()               # and returns to the start
    r.sync()
    g, base = run.grid, r.base[run.rec.ids['arena']]
    grad = {}
    for n in ('th', 'th_a', 'u', 'u_a', 'v', 'v_a', 'w'):
        p = ctypes.c_void_p()
        if r.lib.te_adjoint_device_ptr(r.h, base + run.fields[n] // 4, ctypes.byref(p)):
            raise RuntimeError('no adjoint of ' + n)
        grad[n] = torch.as_tensor(_Words(r, p.value, g.count), device='cuda').view(g.nz + 1, g.strideK, g.strideJ)
    return {'kind': 'adjoint', 'r': r, 'steps': c['steps'], 'every': c['every'], 'grid': g,
            'w': _field(r, run, 'w'), 'grad': grad}


def _members(c):
    """Grids and schedules of an ensemble, in the ranges of scenario.ensemble."""
    rng = random.Random(c['sizes'])
    for _ in range(c['members']):
        nx, ny, nz = 8 * rng.randint(8, 24), 8 * rng.randint(8, 24), 4 * rng.randint(10, 16)
        fine = rng.random() < 0.5
        yield (nx, ny, nz, 500.0 if fine else 1000.0, (12000.0 if fine else 16000.0) / nz, 3.0 if fine else 6.0,
               rng.randint(6, 8), float(rng.randint(10, 30)))


def _prepare_ensemble(c, seed):
    members, outs = [], []
    for m, spec in enumerate(_members(c)):
        run, tape = _run(*spec)
        r = _player(run, tape, seed * 1009 + m, 'fused')
        members.append(r)
        if m < 8:
            outs.append(_outputs(r, run, ('th', 'qv', 'u', 'v', 'w', 'pp3d')))
    return {'kind': 'ensemble', 'ens': Ensemble(members), 'out': outs}


def _prepare_wsolve(c, seed):
    """Column coefficients of the size the acoustic step has them, on fields of our own."""
    nx, ny, nz = c['nx'], c['ny'], c['nz']
    gen = torch.Generator(device='cuda')
    gen.manual_seed(int(seed))
    scale = {'pk1': 2.5e-3, 'pk2': -2.5e-3, 'qk': 2.5e-4, 'mm': 500.0, 'fpk': 1e-5, 'wten': 1e-2, 'pp3d': 1e-4, 'w': 1.0}
    f = {}
    for n, s in scale.items():
        x = torch.rand((nz + 1, ny + 7, nx + 7), generator=gen, device='cuda')
        f[n] = (x.add_(0.5) if n in ('pk1', 'pk2', 'mm') else x.sub_(0.5)).mul_(s)
    args = TeWSolveFields(*[f[n].data_ptr() for n in WSOLVE_IN + ('w',)])
    state = {'kind': 'wsolve', 'f': f, 'args': args, 'dims': (nx, ny, nz), 'lib': load_library()}
    torch.cuda.synchronize()
    return state


DTS, ALPH, BETA = 0.375, 0.6, 0.4


def prepare(case, seed):
    return {'step': _prepare_step, 'physics': _prepare_physics, 'adjoint': _prepare_adjoint,
            'ensemble': _prepare_ensemble, 'wsolve': _prepare_wsolve}[case['kind']](case, seed)


# ------------------------------------------------------------------ one pass


def run(state):
    kind = state['kind']
    if kind == 'step':
        state['r'].encode_steps(1)
        return state['out']
    if kind == 'physics':
        state['r'].encode_steps(state['steps'])
        if state['diag']:
            state['r'].encode_diag()
        return state['out']
    if kind == 'ensemble':
        state['ens'].run(1)
        return state['out']
    if kind == 'adjoint':
        # J = sum of w^2 over the interior at the end of the window; memory returns to the start
        r, g = state['r'], state['grid']
        r.adjoint_forward(state['steps'], state['every'])
        with torch.cuda.stream(_stream()):
            w = state['w'].clone()
            inner = (slice(1, g.nz), slice(3, 3 + g.ny), slice(3, 3 + g.nx))
            torch.mul(w[inner], 2.0, out=state['grad']['w'][inner])
        r.adjoint_backward()
        return {'w': w, 'grad': [state['grad'][n] for n in ('th', 'th_a', 'u', 'u_a', 'v', 'v_a')]}
    f, (nx, ny, nz) = state['f'], state['dims']
    err = ctypes.create_string_buffer(256)
    if state['lib'].te_w_solve_static_scratch(ctypes.byref(state['args']), nx, ny, nz, DTS, ALPH, BETA,
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), err, 256):
        raise RuntimeError(err.value.decode())
    return f['w']


# ------------------------------------------------------------------ what a pass needs


def _step_flops(nsound, variables, nz_points):
    """Operations of a step per point: linear and WENO fluxes with their assembly, substeps,
    and the point-wise kernels around them."""
    substeps = timestep.AcousticSchedule(nsound, 3.0).total
    return nz_points * (2 * variables * 54 + variables * 240 + substeps * 75 + 700)


def work(case):
    kind = case['kind']
    if kind == 'ensemble':
        pts, flops = 0, 0
        for nx, ny, nz, _, _, _, nsound, _ in _members(case):
            pts += (nx + 7) * (ny + 7) * (nz + 1)
            flops += _step_flops(nsound, 5, nx * ny * nz)
        return {'bytes': 4.0 * pts * (29 + 33), 'flops': float(flops)}
    if kind == 'physics':
        nx, ny, nz = {'single_cell': (120, 120, 40), 'squall_line': (300, 60, 40),
                      'supercell_stretched': (144, 144, 40)}[case['recording']]
        # the state is read and written: 12 advected scalars and the winds in two copies, the
        # turbulence and microphysics fields carried from step to step
        return {'bytes': 4.0 * (nx + 7) * (ny + 7) * (nz + 1) * (58 + 64 + (8 if case['diag'] else 0)),
                'flops': float(case['steps'] * (_step_flops(4, 15, nx * ny * nz) + nx * ny * nz * 4000) +
                               (nx * ny * nz * 3000 if case['diag'] else 0))}
    nx, ny, nz = case['nx'], case['ny'], case['nz']
    pts = (nx + 7) * (ny + 7) * (nz + 1)
    if kind == 'wsolve':
        return {'bytes': 4.0 * pts * (len(WSOLVE_IN) + 2), 'flops': 40.0 * nx * ny * nz}
    if kind == 'adjoint':
        # forward, its recomputation and the reverse sweep (about twice a forward)
        return {'bytes': 4.0 * pts * (24 + 7), 'flops': 4.0 * case['steps'] * _step_flops(8, 4, nx * ny * nz)}
    ins, outs = (20, 22) if case['dry'] else (29, 33)
    return {'bytes': 4.0 * pts * (ins + outs), 'flops': float(_step_flops(case['nsound'], 4 if case['dry'] else 5, nx * ny * nz))}


def exact(case, seed):
    """The column solve in 64 bits.  The steps have none here: a 64-bit step of these kernels
    is a model of its own, and in 32 bits its results are fixed to the bit by the tapes."""
    if case['kind'] != 'wsolve':
        return None
    s = _prepare_wsolve(case, seed)
    nx, ny, nz = s['dims']
    box = (slice(None), slice(3, 3 + ny), slice(3, 3 + nx))
    pk1, pk2, qk, mm, fpk, wten, pp = (s['f'][n][box].double() for n in WSOLVE_IN)
    dts, alph, beta = (float(np.float32(x)) for x in (DTS, ALPH, BETA))
    w = s['f']['w'].double()
    w0 = w[box]
    A, B, total, asq = pk1 + qk, pk2 - qk, pp + fpk, alph * alph
    cA, cB = {}, {}
    for k in range(1, nz):
        m = mm[k]
        aa, cc = -asq * m * A[k - 1], asq * m * B[k]
        bb = 1.0 - asq * m * (B[k - 1] - A[k])
        dd = w0[k] + dts * wten[k] - beta * m * (pp[k] - pp[k - 1]) - alph * m * (total[k] - total[k - 1])
        if k > 1:
            bb, dd = bb + aa * cA[k - 1], dd - aa * cB[k - 1]
        cA[k], cB[k] = -cc / bb, dd / bb
    top = cB[nz - 1]
    w[nz - 1][box[1:]] = top
    for k in range(nz - 2, 0, -1):
        top = cA[k] * top + cB[k]
        w[k][box[1:]] = top
    w[0][box[1:]] = 0.0
    w[nz][box[1:]] = 0.0
    return w
