"""Workloads of the Lenia engine, through its public entry points.

Each case is one call a user of the engine makes:

* ``step``   : ``helpers.build_update_fn(...)(rng, state, K, gf, w, dt)``, one
               Euler step (an interactive loop, a per-step training layer);
* ``scan``   : ``runner.run_scan``, a rollout with its whole trajectory
               (rendering a creature, ``init_and_run``);
* ``batch``  : ``runner.run_scan_mem_optimized``, solutions x initial states
               with per-step statistics and the stop counts (a search);
* ``uneven`` : ``batch.UnevenBatch``, worlds of several shapes, radii and
               growth parameters in one captured launch;
* ``grad``   : ``grad.rollout`` with a loss on its last state, forward and
               backward (learning kernels, growth parameters or initial cells).

Worlds are tori of float32 cells.  A search starts from uniform noise in a
central patch, as the benchmark's workloads do; rollouts are short (noise
worlds are chaotic: after some tens of steps two correct float32 programs no
longer agree), every step costs the same whatever the horizon.

``listed`` gives the fixed cases, ``draw`` more of the same ranges, ``prepare``
what a program holds before the call, ``run`` one pass, ``work`` the bytes and
operations that no program can do without, ``exact`` the outputs in 64 bits
from plain torch and numpy.
"""
import math

import numpy as np
import torch

from leniax_gb300 import batch as lbatch
from leniax_gb300 import grad as lgrad
from leniax_gb300 import helpers, kernels, runner, statistics

# shares of the uneven batch's worlds by shape, its radii, growth parameters and time steps
UNEVEN_MIX = (((64, 64), 0.5), ((128, 128), 0.3), ((256, 256), 0.15), ((64, 64, 64), 0.05))
UNEVEN_R, UNEVEN_M, UNEVEN_S, UNEVEN_DT = (5, 26), (0.1, 0.35), (0.03, 0.06), (0.05, 0.1)
EPS = 1e-7
# The statistics that a pass hands back.  The engine computes all twelve every time; the others are counts of cells
# above 1e-7, quotients by such counts, or differences of nearly equal centroids, in which one rounding of a transform
# shows: their tests bound them by cells and by spreads instead.
STATS = ('channel_mass', 'mass', 'growth', 'inertia', 'mass_centroid', 'N', 'N_box')


# ---------------------------------------------------------------- the cases
def case(call, world, sols=1, inits=1, steps=1, channels=1, kernels=1, radius=13.0, dt=0.1, patch=0.375, average=True,
         width=0.03, **more):
    return dict(call=call, world='x'.join(map(str, world)), sols=sols, inits=inits, steps=steps, channels=channels,
                kernels=kernels, radius=radius, dt=dt, patch=patch, average=average, width=width, **more)


def listed():
    return [
        # one interactive step of the single-world model: the smallest call, latency and launches
        dict(case('step', (128, 128)), name='step_128'),
        # one step of a handful of three-channel worlds whose side is no power of two
        dict(case('step', (100, 100), inits=8, channels=3, kernels=9, radius=12.0, dt=0.2), name='step_100_c3k9'),
        # a three-channel, fifteen-kernel creature played with all its states, fields and potentials kept
        dict(case('scan', (128, 128), steps=32, channels=3, kernels=15, radius=12.0, dt=0.2, average=False),
             name='scan_128_c3k15'),
        # the search batch: a thousand noise worlds of one model with statistics and both stop counts
        dict(case('batch', (128, 128), inits=1024, steps=6, width=0.015), name='search_128'),
        # a generation of a quality-diversity search: every solution with its own growth and several initial states
        dict(case('batch', (64, 64), sols=96, inits=8, steps=12), name='generation_64'),
        # the multi-channel batch
        dict(case('batch', (256, 256), inits=256, steps=16, channels=3, kernels=15, radius=20.0, dt=0.2),
             name='batch_256_c3k15'),
        # a search on worlds whose side is no power of two
        dict(case('batch', (100, 100), inits=256, steps=12), name='search_100'),
        # 3D worlds that no power of two fits
        dict(case('batch', (48, 48, 48), inits=64, steps=10, radius=8.0, patch=1 / 3), name='batch_48cube'),
        # one large world, watched at high resolution
        dict(case('batch', (1024, 1024), inits=2, steps=8, radius=52.0), name='large_1024'),
        # the uneven search: 4096 worlds of four shapes, each with its own radius, growth and time step
        dict(case('uneven', (0, ), inits=4096, steps=5, patch=1 / 3), name='uneven_4096'),
        # learning a kernel, growth parameters and initial cells of the single-world model on a batch
        dict(case('grad', (128, 128), inits=64, steps=8, average=False, ckpt=4), name='grad_128'),
        # the same for one 3D world
        dict(case('grad', (48, 48, 48), steps=12, radius=8.0, patch=1 / 3, average=False, ckpt=4),
             name='grad_48cube'),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side2d(rng, lo, hi):
    """A world side: powers of two, the even sides configurations use, and any other number."""
    kind = rng.random()
    if kind < 0.4:
        return 2**rng.randint(math.ceil(math.log2(lo)), int(math.log2(hi)))
    side = _log(rng, lo, hi)
    if kind < 0.8:  # of factors 2, 3, 5, 7
        while True:
            n = side
            for p in (2, 3, 5, 7):
                while n % p == 0:
                    n //= p
            if n == 1:
                return side
            side -= 1
    return side


def _model(rng):
    """(channels, kernels, average)"""
    return rng.choice([(1, 1, True), (1, 1, True), (1, 2, True), (2, 2, True), (3, 9, True), (3, 15, False)])


def draw(rng):
    call = rng.choice(['step', 'scan', 'batch', 'batch', 'batch', 'batch3d', 'large', 'uneven', 'grad', 'grad3d'])
    C, K, avg = _model(rng)
    dt = 0.1 if K == 1 else rng.choice([0.1, 0.2])
    if call == 'uneven':
        return case('uneven', (0, ), inits=_log(rng, 128, 4096), steps=rng.randint(3, 5), patch=1 / 3)
    if call in ('batch3d', 'grad3d'):
        side = rng.choice([24, 27, 32, 36, 40, 45, 48, 56, 64])
        world = (side, side, side) if rng.random() < 0.75 else (side, 40, 36)
        cells = math.prod(world)
        top = 64 * 48**3 if call == 'batch3d' else 4 * 48**3
        n = max(1, min(_log(rng, 1, 64), top // cells))
        if call == 'grad3d':
            return case('grad', world, inits=n, steps=rng.randint(4, 12), radius=float(rng.randint(5, 8)), patch=1 / 3,
                        average=False, ckpt=4)
        return case('batch', world, inits=n, steps=rng.randint(4, 10), radius=float(rng.randint(5, 8)), patch=1 / 3)
    if call == 'large':
        side = _side2d(rng, 512, 1024)
        return case('batch', (side, side), inits=rng.randint(1, 2), steps=rng.randint(4, 8),
                    radius=float(rng.randint(13, 52)))
    side = _side2d(rng, 32, 256)
    world = (side, side) if rng.random() < 0.75 else (side, _side2d(rng, 32, 256))
    radius = float(rng.randint(5, max(5, min(20, min(world) // 3))))
    units = math.prod(world) * (C + K)  # of one world's step
    if call == 'step':
        n = max(1, min(_log(rng, 1, 32), 16 * 256 * 256 * 4 // units))
        return case('step', world, inits=n, channels=C, kernels=K, radius=radius, dt=dt, average=avg)
    if call == 'scan':
        n = max(1, min(_log(rng, 1, 8), 2 * 128 * 128 * 18 // units))
        return case('scan', world, inits=n, steps=rng.randint(4, 32 if K > 1 else 12), channels=C, kernels=K,
                    radius=radius, dt=dt, average=avg)
    if call == 'grad':
        n = max(1, min(_log(rng, 1, 64), 64 * 128 * 128 * 2 // units))
        return case('grad', world, inits=n, steps=rng.randint(4, 8), channels=C, kernels=K, radius=radius, dt=dt,
                    average=avg and K > 1, ckpt=4)
    sols = rng.choice([1, 1, 1, 4, 16])
    n = max(1, min(_log(rng, 8, 1024), 1024 * 128 * 128 * 2 // units) // sols)
    return case('batch', world, sols=sols, inits=n, steps=rng.randint(4, 12), channels=C, kernels=K, radius=radius,
                dt=dt, average=avg)


# ---------------------------------------------------------------- inputs
def _world(c):
    return tuple(int(v) for v in c['world'].split('x'))


def _device():
    return torch.device('cuda', torch.cuda.current_device())


def _generator(seed, offset=0):
    return torch.Generator(_device()).manual_seed(1000 * seed + offset)


def _patches(n, C, world, share, gen):
    """``[n, C, *world]``: uniform noise in a central patch, scaled by a per-world factor in [0.5, 1]."""
    p = [max(2, int(round(w * share))) for w in world]
    cells = torch.zeros((n, C) + tuple(world), device=gen.device)
    noise = torch.rand((n, C) + tuple(p), generator=gen, device=gen.device)
    factor = 0.5 + 0.5 * torch.rand((n, ) + (1, ) * (1 + len(world)), generator=gen, device=gen.device)
    at = tuple(slice((w - q) // 2, (w - q) // 2 + q) for w, q in zip(world, p))
    cells[(slice(None), slice(None)) + at] = noise * factor
    return cells


def _target(c):
    """``[C, *world]``: what a learned creature should become, a smooth ball in the middle of every channel."""
    axes = [(torch.arange(w, dtype=torch.float64, device=_device()) - w // 2) / (c['patch'] * w / 2)
            for w in _world(c)]
    ball = torch.exp(-sum(g**2 for g in torch.meshgrid(*axes, indexing='ij')))
    return 0.5 * ball.expand((c['channels'], ) + ball.shape)


def _kernels_params(c):
    """leniax's kernels_params of the case's model: the one-kernel bump model, or a seeded kernel set as in the
    multi-channel workload."""
    C, nk = c['channels'], c['kernels']
    if nk == 1:
        return [{'k_slug': 'circle_2d', 'k_params': [1.0, [1.0]], 'kf_slug': 'gauss_bump', 'kf_params': [1.0],
                 'gf_slug': 'gaussian', 'gf_params': [0.15, c['width']], 'h': 1.0, 'c_in': 0,
                 'c_out': 0}]
    rng = np.random.Generator(np.random.PCG64(nk))
    out = []
    for k in range(nk):
        b = [float(x) for x in rng.random(int(rng.integers(1, 4)))]
        b[int(np.argmax(b))] = 1.0
        out.append({'k_slug': 'circle_2d', 'k_params': [float(rng.uniform(0.5, 1.0)), b], 'kf_slug': 'gauss_bump',
                    'kf_params': [1.0], 'gf_slug': 'gaussian',
                    'gf_params': [float(rng.uniform(0.1, 0.4)), float(rng.uniform(0.04, 0.16))],
                    'h': float(rng.uniform(0.1, 1.0)), 'c_in': k * C // nk,
                    'c_out': k % C})
    for ch in range(C):
        total = sum(p['h'] for p in out if p['c_out'] == ch)
        for p in out:
            if p['c_out'] == ch:
                p['h'] /= total
    return out


def _growths(c, seed):
    """``[sols, K, 2]``: the model's growth parameters, one solution's differing from the next by some per cent."""
    base = torch.tensor([p['gf_params'] for p in _kernels_params(c)], device=_device())
    if c['sols'] == 1:
        return base[None].contiguous()
    jitter = torch.rand((c['sols'], ) + tuple(base.shape), generator=_generator(seed, 1), device=_device())
    return base * (0.95 + 0.1 * jitter)


def _uneven_inputs(c, seed):
    """Per shape: (world, cells ``[n, *world]``, R ``[n]``, gf ``[n, 2]``, dt ``[n]``)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for i, (world, share) in enumerate(UNEVEN_MIX):
        n = max(1, int(round(c['inits'] * share)))
        cells = _patches(n, 1, world, c['patch'], _generator(seed, i))[:, 0]
        R = rng.integers(UNEVEN_R[0], UNEVEN_R[1] + 1, size=n).astype(np.float32)
        gf = np.stack([rng.uniform(*UNEVEN_M, size=n), rng.uniform(*UNEVEN_S, size=n)], 1).astype(np.float32)
        dt = rng.choice(np.asarray(UNEVEN_DT), size=n)
        out.append((world, cells, R, gf, dt))
    return out


def prepare(c, seed):
    dev = _device()
    if c['call'] == 'uneven':
        ring = _kernels_params(case('batch', (64, 64)))[0]
        classes = []
        for world, cells, R, gf, dt in _uneven_inputs(c, seed):
            classes.append(lbatch.WorldClass(cells0=cells, K=lbatch.world_spectra(world, R, ring, dev),
                                             gf_params=torch.from_numpy(gf).to(dev),
                                             weights=torch.ones(len(R), device=dev),
                                             T=torch.from_numpy((1.0 / dt).astype(np.float32)).to(dev),
                                             R=torch.from_numpy(R).to(dev)))
        return {'case': c, 'batch': lbatch.UnevenBatch(classes, c['steps']).capture()}
    world = _world(c)
    C, sols, inits = c['channels'], c['sols'], c['inits']
    K, mapping = kernels.get_kernels_and_mapping(_kernels_params(c), list(world), C, c['radius'], True, dev)
    s = {'case': c, 'update': helpers.build_update_fn(K.shape, mapping, 'v1', c['average']),
         'stats': statistics.ComputeStatsFn(world, c['radius'], 1.0 / c['dt']),
         'w': mapping.get_kernels_weight_per_channel(dev), 'gf': _growths(c, seed)}
    cells = _patches(sols * inits, C, world, c['patch'], _generator(seed))
    if c['call'] in ('step', 'scan'):
        s.update(cells=cells, K=K, gf=s['gf'][0], T=torch.tensor(1.0 / c['dt'], device=dev))
    elif c['call'] == 'batch':
        s.update(cells=cells.reshape((sols, inits, C) + world), K=K[None].expand((sols, ) + K.shape).contiguous(),
                 w=s['w'][None].expand((sols, ) + s['w'].shape).contiguous(),
                 T=torch.full((sols, ), 1.0 / c['dt'], device=dev))
    else:
        s.update(cells=cells[None], target=_target(c).float()[None, None], w=s['w'][None], T=torch.tensor([1.0 / c['dt']], device=dev),
                 k_real=_world_kernels(c).float().to(dev)[None])
    return s


def _kept(stats):
    return {k: stats[k] for k in STATS if k in stats}


def run(s):
    c = s['case']
    if c['call'] == 'step':
        return s['update'](None, s['cells'], s['K'], s['gf'], s['w'], c['dt'])
    if c['call'] == 'scan':
        *trajectory, stats = runner.run_scan(None, s['cells'], s['K'], s['gf'], s['w'], s['T'], c['steps'],
                                             c['radius'], s['update'], s['stats'])
        return trajectory, _kept(stats)
    if c['call'] == 'batch':
        stats, final = runner.run_scan_mem_optimized(None, s['cells'], s['K'], s['gf'], s['w'], s['T'], c['steps'],
                                                     c['radius'], s['update'], s['stats'], with_box=True,
                                                     with_centroid=True)
        return _kept(stats), final
    if c['call'] == 'uneven':
        return [(_kept(r['stats']), r['final']) for r in s['batch'].run().results()]
    leaves = [s[k].detach().requires_grad_(True) for k in ('cells', 'k_real', 'gf', 'w')]
    final = lgrad.rollout(*leaves, s['T'], s['update'], c['steps'], c['ckpt'])
    loss = ((final - s['target'])**2).mean()
    return {'loss': loss.detach(), 'final': final.detach(), 'grads': torch.autograd.grad(loss, leaves)}


# ---------------------------------------------------------------- what a pass cannot do without
def _step_flops(C, K, P, stats):
    """Real transforms of every channel and kernel, the spectrum product, growth, weighting, update, statistics."""
    f = (C + K) * 2.5 * P * math.log2(P) + 6 * K * (P // 2 + 1) + 10 * K * P + 4 * C * P
    return f + (10 * C * P if stats else 0)


def work(c):
    if c['call'] == 'uneven':
        b = f = 0
        for world, share in UNEVEN_MIX:
            n, P, nd = max(1, int(round(c['inits'] * share))), math.prod(world), len(world)
            f += n * c['steps'] * _step_flops(1, 1, P, True)
            b += n * (4 * 2 * P + 8 * math.prod(world[:-1]) * (world[-1] // 2 + 1) + c['steps'] * 4 * (12 + nd))
        return {'bytes': b, 'flops': f}
    world = _world(c)
    C, K, P, n, steps = c['channels'], c['kernels'], math.prod(world), c['sols'] * c['inits'], c['steps']
    spectrum = 8 * K * math.prod(world[:-1]) * (world[-1] // 2 + 1)
    if c['call'] == 'step':
        return {'bytes': n * 4 * P * (3 * C + K) + spectrum, 'flops': n * _step_flops(C, K, P, False)}
    flops = n * steps * _step_flops(C, K, P, True)
    if c['call'] == 'scan':
        return {'bytes': n * 4 * P * (C + steps * (2 * C + K)) + n * steps * 4 * (C + 11) + spectrum, 'flops': flops}
    if c['call'] == 'batch':
        return {'bytes': n * 4 * P * 2 * C + n * steps * 4 * (C + 11 + len(world)) + c['sols'] * spectrum,
                'flops': flops}
    # forward and reverse: the reverse step transforms dL/du of every kernel, the states and the correlations
    reverse = (2 * C + K) * 2.5 * P * math.log2(P) + 14 * K * (P // 2 + 1) + 20 * K * P
    return {'bytes': n * 4 * P * 4 * C + 2 * 4 * K * P, 'flops': n * steps * (_step_flops(C, K, P, False) + reverse)}


# ---------------------------------------------------------------- the outputs in 64 bits
def _ring(R, k_params, world):
    """World-sized ring kernel as leniax places it (kernels.py:93-148), float64 on the host: the bump
    ``exp(1 - 1/(x(1 - x) + 1e-7))`` over each ring of ``k_params`` = [relative radius, ring weights]."""
    r, b = k_params[0], np.asarray(k_params[1])
    k = math.ceil(r * R)
    grid = np.meshgrid(*[(np.arange(2 * k) - k) / (r * R)] * len(world), indexing='ij')
    d = np.sqrt(sum(g**2 for g in grid))
    x = np.mod(len(b) * d, 1.0)
    with np.errstate(over='ignore', under='ignore'):
        ring = np.exp(1 - 1 / (x * (1 - x) + EPS)) * b[np.minimum(np.floor(len(b) * d).astype(int), len(b) - 1)]
    ring = np.where(d < 1, ring, 0)
    full = np.zeros(world)
    # centred in the world, then shifted by half of it: the centre of an odd side ends at its last index
    at = tuple(((w - 2 * k) // 2 + np.arange(2 * k) + w // 2) % w for w in world)
    np.add.at(full, np.ix_(*at), ring / ring.sum())
    return torch.from_numpy(full)


def _world_kernels(c):
    """``[K, *world]`` float64: the model's kernels in the order of their input channels."""
    return torch.stack([_ring(c['radius'], p['k_params'], _world(c)) for p in _kernels_params(c)])


def _tables(c):
    kp = _kernels_params(c)
    w = torch.zeros(c['channels'], len(kp), dtype=torch.float64, device=_device())
    for k, p in enumerate(kp):
        w[p['c_out'], k] = p['h']
    return [p['c_in'] for p in kp], w


def _step64(cells, kh, cin, gf, w, dt, average):
    """(new cells before the clip, field, potential) of ``cells`` ``[n, C, *world]``; ``kh`` ``[1 or n, K, *half]``,
    ``gf`` ``[1 or n, K, 2]``, ``w`` ``[C, K]``, ``dt`` a number or ``[n]``."""
    nd = cells.dim() - 2
    axes = tuple(range(-nd, 0))
    spec = torch.fft.rfftn(cells, dim=axes)[:, cin] * kh
    pot = torch.fft.irfftn(spec, s=cells.shape[2:], dim=axes)
    m, s = (gf[..., i].reshape(gf.shape[:2] + (1, ) * nd) for i in (0, 1))
    g = 2 * torch.exp(-((pot - m) / s)**2 / 2) - 1
    field = torch.einsum('ck,nk...->nc...', w, g)
    if average:
        field = field / w.sum(1).reshape((1, -1) + (1, ) * nd)
    if torch.is_tensor(dt):
        dt = dt.reshape((-1, ) + (1, ) * (1 + nd))
    return cells + dt * field, field, pot


class _Stats64:
    """The kept statistics of ``n`` worlds over a rollout: masses, positive growth, moment of inertia and centroid in
    the carried centred frame, and the two stop counts."""

    def __init__(self, n, world, R, dev):
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=dev)  # noqa: E731
        self.world, self.R2, self.n = world, R * R, n
        self.shift, self.first, self.rows = z(n, len(world)), None, []
        self.go, self.go_box, self.N, self.N_box = z(n) + 1, z(n) + 1, z(n), z(n)

    def add(self, cells, field):
        nd = len(self.world)
        every = tuple(range(1, 2 + nd))
        m0 = cells.sum(every)
        channel = cells.sum(every[1:]) / (self.R2[:, None] if torch.is_tensor(self.R2) else self.R2)
        first, second = [], []
        for ax, size in enumerate(self.world):
            line = cells.sum(dim=[1] + [2 + i for i in range(nd) if i != ax])
            p = torch.arange(size, device=cells.device, dtype=torch.float64)
            at = torch.remainder(p[None] - self.shift[:, ax:ax + 1], size) - size // 2
            first.append((line * at).sum(1))
            second.append((line * at**2).sum(1))
        mx, mx2 = torch.stack(first, 1), torch.stack(second, 1)
        cen = mx / (m0 + EPS)[:, None]
        size = torch.tensor(self.world, dtype=torch.float64, device=cells.device)
        self.rows.append({'channel_mass': channel, 'mass': m0 / self.R2,
                          'growth': field.clamp(min=0).sum(every) / self.R2,
                          'inertia': ((mx2 - cen * mx) / (m0**2 + EPS)[:, None]).sum(1),
                          'mass_centroid': torch.remainder(cen + torch.floor(size / 2) + self.shift, size)})
        self.shift = torch.remainder(self.shift + cen.trunc(), size)
        # horizons are shorter than the 128 steps after which a monotone or large mass stops a world
        self.first = channel if self.first is None else self.first
        self.go = self.go * ((channel >= EPS) & (channel <= 3 * self.first)).all(1)
        edge = torch.zeros(self.n, dtype=torch.bool, device=cells.device)
        for ax in range(nd):
            for at in (0, self.world[ax] - 1):
                edge |= (cells.select(2 + ax, at) > EPS).flatten(1).any(1)
        self.go_box = self.go_box * ((m0 >= 1e-3) & (m0 <= 0.9 * cells[0].numel()) & ~edge)
        self.N, self.N_box = self.N + self.go, self.N_box + self.go_box

    def result(self, sols):
        """The dict that run() returns: ``[sols, T, inits, ...]``, the counts ``[sols, inits]``."""
        out = {k: torch.stack([r[k] for r in self.rows]) for k in self.rows[0]}
        out = {k: v.reshape((v.shape[0], sols, -1) + tuple(v.shape[2:])).transpose(0, 1) for k, v in out.items()}
        out['N'], out['N_box'] = self.N.reshape(sols, -1), self.N_box.reshape(sols, -1)
        return out


def _chunks(n, values):
    """Slices of ``n`` worlds of ``values`` 64-bit values each that stay within a few GB."""
    step = max(1, int(2.5e8 / values))
    return [slice(i, min(n, i + step)) for i in range(0, n, step)]


def _half(full):
    return torch.fft.rfftn(full, dim=tuple(range(1, full.dim())))


def _rollout64(c, cells, kh, cin, gf, w, dt, R, world, keep=None):
    """(final cells, statistics of every chunk of worlds); ``gf`` and ``kh`` one row for all or one per world."""
    finals, stats = [], []
    C, K = cells.shape[1], gf.shape[1]
    of = lambda t, at: t[at] if torch.is_tensor(t) and t.shape[0] == cells.shape[0] > 1 else t  # noqa: E731
    for at in _chunks(cells.shape[0], math.prod(world) * (C + 4 * K)):
        x = cells[at].double()
        st = _Stats64(x.shape[0], world, of(R, at), x.device)
        for _ in range(c['steps']):
            new, field, pot = _step64(x, of(kh, at), cin, of(gf, at), w, of(dt, at), c['average'])
            st.add(x, field)
            if keep is not None:
                keep.append((x, field, pot))
            x = new.clamp(0, 1)
        finals.append(x)
        stats.append(st)
    return torch.cat(finals), stats


def _joined(stats, sols):
    """One _Stats64 of several chunks' worlds."""
    all_ = stats[0]
    if len(stats) > 1:
        all_.rows = [{k: torch.cat([s.rows[t][k] for s in stats]) for k in stats[0].rows[0]}
                     for t in range(len(stats[0].rows))]
        all_.N, all_.N_box = torch.cat([s.N for s in stats]), torch.cat([s.N_box for s in stats])
    return all_.result(sols)


def exact(c, seed):
    dev = _device()
    if c['call'] == 'uneven':
        out = []
        k_params = _kernels_params(case('batch', (64, 64)))[0]['k_params']
        for world, cells, R, gf, dt in _uneven_inputs(c, seed):
            # the same radii recur: one kernel for each
            radii = sorted(set(R.tolist()))
            table = _half(torch.stack([_ring(r, k_params, world) for r in radii]).to(dev))
            row = torch.tensor([radii.index(r) for r in R.tolist()], device=dev)
            gft = torch.from_numpy(gf).to(dev).double()[:, None]
            dtt, Rt = (torch.from_numpy(np.asarray(v, np.float64)).to(dev) for v in (dt, R))
            one = torch.ones((1, 1), dtype=torch.float64, device=dev)
            parts = []
            for at in _chunks(len(R), math.prod(world) * 5):
                parts.append(_rollout64(c, cells[at, None], table[row[at]][:, None], [0], gft[at], one, dtt[at], Rt[at],
                                        world))
            st = _joined([s for _, p in parts for s in p], len(R))
            out.append((st, torch.cat([f for f, _ in parts])[:, 0]))
        return out
    world = _world(c)
    C, sols, inits = c['channels'], c['sols'], c['inits']
    cin, w = _tables(c)
    w = w.float().double()
    cells = _patches(sols * inits, C, world, c['patch'], _generator(seed))
    gf = _growths(c, seed).double()
    kern = _world_kernels(c).float().double().to(dev)
    if c['call'] == 'grad':
        return _grads64(c, cells, kern, cin, gf, w)
    kh = _half(kern)[None]
    if c['call'] == 'step':
        new, field, pot = _step64(cells.double(), kh, cin, gf, w, c['dt'], c['average'])
        return new.clamp(0, 1), field, pot
    gf = gf.repeat_interleave(inits, 0) if sols > 1 else gf
    keep = [] if c['call'] == 'scan' else None
    final, stats = _rollout64(c, cells, kh, cin, gf, w, c['dt'], c['radius'], world, keep)
    st = _joined(stats, sols)
    if keep is not None:
        st = {k: v[0] for k, v in st.items() if k not in ('N_box', 'mass_centroid')}
        return [torch.stack([x[i] for x in keep]) for i in range(3)], st
    return st, final.reshape((sols, inits, C) + world)


def _grads64(c, cells, kern, cin, gf, w):
    """Loss, last state and gradients; worlds add up in the kernel's, the growth parameters' and the weights'."""
    world, C, n = _world(c), c['channels'], c['inits']
    target = _target(c).float().double()[None]
    loss, finals, g_cells, shared = 0.0, [], [], None
    for at in _chunks(n, math.prod(world) * (2 * C + 8 * c['kernels']) * c['steps']):
        x0 = cells[at].double().requires_grad_(True)
        leaves = [t.detach().clone().requires_grad_(True) for t in (kern, gf, w)]
        kh = _half(leaves[0])[None]
        x = x0
        for _ in range(c['steps']):
            pre = _step64(x, kh, cin, leaves[1], leaves[2], c['dt'], c['average'])[0]
            # leniax's clip passes gradients straight through.  (The mask form is discontinuous: a cell within a
            # rounding of a bound has one gradient or another, so it is left to its tests.)
            x = pre + (pre.clamp(0, 1) - pre).detach()
        part = ((x - target)**2).sum() / cells.numel()
        g = torch.autograd.grad(part, [x0] + leaves)
        loss = loss + part.detach()
        finals.append(x.detach())
        g_cells.append(g[0])
        shared = list(g[1:]) if shared is None else [a + b for a, b in zip(shared, g[1:])]
    return {'loss': loss, 'final': torch.cat(finals)[None],
            'grads': (torch.cat(g_cells)[None], shared[0][None], shared[1], shared[2][None])}
