"""Performance cases of the turn loop: what a user of this package has it do.

Every case is one pass through the public classes (Particles, the element
lists, TurnGraph, BatchedTurn, the slicers and statistics) on a matched 6D
Gaussian bunch at 26 GeV/c in a 6.9 km ring.  Bunches carry a tenth of the
nominal intensity so that a state that is tracked for thousands of passes
stays far from the exponential growth of an unstable bunch.

Kinds of case:

* ``graph``   a captured turn (or a full ring of the multi-turn wake)
              replayed: [TransverseMap, RFSystems | LinearMap, WakeField].
* ``eager``   the user's own loop, one turn, bunch-dependent cuts and a
              damper, then the centroid and all coordinates.
* ``charge``  one eager turn with uniform-charge slices and the dipolar and
              quadrupolar wakes of parallel plates.
* ``batch``   many bunches of uneven size in one persistent launch a turn.
* ``monitor`` the maps of one turn without wakes, then the bunch statistics
              a monitor stores.
* ``slices``  a slice set with every per-slice statistic.
"""
import random

import numpy as np
import torch
from scipy.constants import c, e, m_p

C_RING = 6911.5038378975451
GAMMA = 27.7
Q_X, Q_Y, Q_S, BETA = 20.13, 20.18, 0.017, 50.
Z_CUTS = (-0.69, 0.69)
ALPHA_C = 230. * 2 * np.pi * Q_S / C_RING + GAMMA**-2
HARMONIC, VOLTAGE = 4620, 4.5e6
CHROMA = (5., 5.)
AMPLITUDE = (1e-11, 1e-11, -5e-12)
SIGMA_Z, SIGMA_DP, EPSN = 0.23, 1e-3, 2.5e-6
INTENSITY = 2.5e10
RESONATOR = (10e6, 1e9, 1.)
WALL = (0.02, C_RING, 5.8e7, 1e-12)
DAMPING = 50.
BATCH_TURNS = 10
COORDS = ('x', 'xp', 'y', 'yp', 'z', 'dp')
BUNCH_STATS = ('mean_x', 'mean_xp', 'mean_y', 'mean_yp', 'mean_z', 'mean_dp',
               'sigma_x', 'sigma_y', 'sigma_z', 'sigma_dp', 'epsn_x',
               'epsn_y', 'epsn_z')
SLICE_STATS = ('mean_x', 'mean_y', 'mean_z', 'mean_xp', 'mean_yp', 'mean_dp',
               'sigma_x', 'sigma_y', 'sigma_z', 'sigma_dp', 'epsn_x',
               'epsn_y', 'epsn_z')
SLICE_CUTS = (-0.46, 0.46)


def listed():
    return [
        # a quick stability check: linear maps, few slices, one resonator;
        # a turn is so short that launches and latency count
        dict(name='linear_f64', kind='graph', form='fp64', n=100000,
             slices=50, detuned=False, rf=False, wake_turns=1),
        # Landau damping studies: chromaticity and octupoles, RF bucket
        dict(name='detuned_f64', kind='graph', form='fp64', n=1000000,
             slices=200, detuned=True, rf=True, wake_turns=1),
        dict(name='detuned_f32', kind='graph', form='fp32', n=1000000,
             slices=200, detuned=True, rf=True, wake_turns=1),
        # growth rates with a resistive wall that is remembered for 50 turns
        dict(name='wall50_f64', kind='graph', form='fp64', n=10000000,
             slices=500, detuned=False, rf=True, wake_turns=50),
        dict(name='wall50_f32', kind='graph', form='fp32', n=10000000,
             slices=500, detuned=False, rf=True, wake_turns=50),
        # the largest bunch: slow headtail modes need a low noise floor
        dict(name='large_f32', kind='graph', form='fp32', n=50000000,
             slices=1000, detuned=True, rf=True, wake_turns=50),
        # scans over chromaticity and intensity
        dict(name='batch_f32', kind='batch', form='fp32', bunches=64,
             smallest=10000, largest=1000000, slices=100),
        dict(name='batch_f64', kind='batch', form='fp64', bunches=24,
             smallest=10000, largest=300000, slices=100),
        # the plain user loop of a machine with a damper, cuts following the
        # bunch, the centroid logged every turn; an odd bunch size
        dict(name='eager_f64', kind='eager', form='fp64', n=100003,
             slices=200),
        # parallel plates with uniform-charge slices
        dict(name='charge_f64', kind='charge', form='fp64', n=50000,
             slices=500),
        # emittance growth without wakes: maps and a full set of statistics
        dict(name='monitor_f64', kind='monitor', form='fp64', n=3000001,
             detuned=True),
        # headtail pictures: every statistic of every slice
        dict(name='slices_f64', kind='slices', form='fp64', n=1000000,
             slices=200),
    ]


def _log_int(rng, lo, hi):
    v = int(round(10 ** rng.uniform(np.log10(lo), np.log10(hi))))
    return max(lo, min(hi, v))


def draw(rng):
    kind = rng.choice(['graph', 'graph', 'graph', 'graph', 'graph', 'batch',
                       'eager', 'charge', 'monitor', 'slices'])
    form = rng.choice(['fp64', 'fp32'])
    if kind == 'graph':
        detuned = rng.random() < 0.5
        turns = rng.choice([1, 1, 1, 2, 10, 50])
        # an FP64 detuned turn costs several times an undetuned one
        top = 10000000 if not detuned or form == 'fp32' \
            else min(10000000, 100000000 // turns)
        return dict(kind='graph', form=form, n=_log_int(rng, 10000, top),
                    slices=_log_int(rng, 20, 1000), detuned=detuned,
                    rf=rng.random() < 0.75, wake_turns=turns)
    if kind == 'batch':
        return dict(kind='batch', form=form, bunches=rng.randint(4, 24),
                    smallest=rng.choice([1001, 10000]),
                    largest=_log_int(rng, 20000, 300000),
                    slices=_log_int(rng, 20, 200))
    if kind == 'eager':
        return dict(kind='eager', form='fp64', n=_log_int(rng, 10000, 1000000),
                    slices=_log_int(rng, 50, 500))
    if kind == 'charge':
        return dict(kind='charge', form='fp64', n=_log_int(rng, 50000, 500000),
                    slices=_log_int(rng, 50, 500))
    if kind == 'monitor':
        return dict(kind='monitor', form=form, n=_log_int(rng, 10000, 10000000),
                    detuned=rng.random() < 0.5)
    slices = _log_int(rng, 20, 500)
    return dict(kind='slices', form='fp64',
                n=_log_int(rng, 1000 * slices, 1000000), slices=slices)


# ------------------------------------------------------------------ inputs

def _coordinates(n, seed, form, device='cuda'):
    """The matched Gaussian bunch of this seed in the form's precision."""
    g = torch.Generator(device=device).manual_seed(int(seed))
    eps = EPSN / np.sqrt(GAMMA**2 - 1)
    sigmas = {'x': np.sqrt(eps * BETA), 'xp': np.sqrt(eps / BETA),
              'y': np.sqrt(eps * BETA), 'yp': np.sqrt(eps / BETA),
              'z': SIGMA_Z, 'dp': SIGMA_DP}
    dt = torch.float64 if form == 'fp64' else torch.float32
    return {k: (torch.randn(n, generator=g, device=device,
                            dtype=torch.float64) * s).to(dt)
            for k, s in sigmas.items()}


def _batch_draws(case, seed):
    """The sizes belong to the case, what is scanned to the seed."""
    rs = np.random.RandomState(3)
    sizes = np.round(10 ** rs.uniform(np.log10(case['smallest']),
                                      np.log10(case['largest']),
                                      size=case['bunches'])).astype(int)
    rs = np.random.RandomState(seed % (1 << 31))
    return (sizes, rs.uniform(-5., 15., size=case['bunches']),
            rs.uniform(5e9, 2e10, size=case['bunches']))


# ------------------------------------------------------------- the package

def _beam(n, intensity, coords, form):
    from pyheadtail_gb300.particles.particles import Particles
    return Particles(n, intensity / n, e, m_p, C_RING, GAMMA,
                     coords_n_momenta_dict=coords, precision=form)


def _printers():
    from pyheadtail_gb300.general.printers import SilentPrinter
    sp = SilentPrinter()
    return dict(printer=sp, warningprinter=sp)


def _transverse(chroma, amplitude):
    from pyheadtail_gb300.trackers.detuners import (AmplitudeDetuning,
                                                    Chromaticity)
    from pyheadtail_gb300.trackers.transverse_tracking import TransverseMap
    detuners = []
    if chroma is not None:
        detuners.append(Chromaticity(*chroma))
    if amplitude is not None:
        detuners.append(AmplitudeDetuning(*amplitude))
    z2, b2 = np.zeros(2), np.array([BETA, BETA])
    return list(TransverseMap(np.array([0., C_RING]), z2, b2, z2, z2, b2, z2,
                              Q_X, Q_Y, detuners, **_printers()))


def _longitudinal(rf):
    from pyheadtail_gb300.trackers.longitudinal_tracking import (LinearMap,
                                                                 RFSystems)
    if rf:
        return RFSystems(C_RING, [HARMONIC], [VOLTAGE], [0.], [ALPHA_C],
                         GAMMA, charge=e, mass=m_p, **_printers())
    return LinearMap([ALPHA_C], C_RING, Q_S, **_printers())


def _bin_slicer(n_slices, **cuts):
    from pyheadtail_gb300.particles.slicing import UniformBinSlicer
    return UniformBinSlicer(n_slices, **cuts, **_printers())


def _wakes(slicer, wake_turns):
    from pyheadtail_gb300.impedances import wakes as W
    sources = [W.CircularResonator(*RESONATOR)]
    if wake_turns > 1:
        sources.append(W.CircularResistiveWall(*WALL, n_turns_wake=wake_turns))
    return W.WakeField(slicer, *sources)


def _warmup(case):
    """Eager turns before the capture: the wake history fills, the host
    scalars settle."""
    return case['wake_turns'] + 5


def prepare(case, seed):
    kind = case['kind']
    if kind == 'batch':
        return _prepare_batch(case, seed)
    coords = _coordinates(case['n'], seed, case['form'])
    beam = _beam(case['n'], INTENSITY, coords, case['form'])
    s = dict(kind=kind, beam=beam, form=case['form'])
    if kind == 'graph':
        from pyheadtail_gb300.turngraph import TurnGraph
        detuned = case['detuned']
        elements = _transverse(CHROMA if detuned else None,
                               AMPLITUDE if detuned else None)
        elements += [_longitudinal(case['rf']),
                     _wakes(_bin_slicer(case['slices'], z_cuts=Z_CUTS),
                            case['wake_turns'])]
        s['turn'] = TurnGraph(elements, beam,
                              warmup_turns=_warmup(case)).capture()
    elif kind == 'eager':
        from pyheadtail_gb300.feedback.transverse_damper import \
            TransverseDamper
        s['elements'] = _transverse((2., 2.), None) + [
            _longitudinal(True),
            TransverseDamper(DAMPING, DAMPING, **_printers()),
            _wakes(_bin_slicer(case['slices'], n_sigma_z=3), 1)]
    elif kind == 'charge':
        from pyheadtail_gb300.impedances import wakes as W
        from pyheadtail_gb300.particles.slicing import UniformChargeSlicer
        random.seed(int(seed))
        slicer = UniformChargeSlicer(case['slices'], n_sigma_z=3,
                                     **_printers())
        s['elements'] = _transverse(None, None) + [
            _longitudinal(True),
            W.WakeField(slicer, W.ParallelPlatesResistiveWall(*WALL))]
    elif kind == 'monitor':
        detuned = case['detuned']
        s['elements'] = _transverse(CHROMA if detuned else None,
                                    AMPLITUDE if detuned else None)
        s['elements'].append(_longitudinal(True))
    else:
        s['slicer'] = _bin_slicer(case['slices'], z_cuts=SLICE_CUTS)
    return s


def _prepare_batch(case, seed):
    from pyheadtail_gb300.batch import BatchedTurn, BunchBatch
    sizes, chroma, intensity = _batch_draws(case, seed)
    beams, maps = [], []
    for b, n in enumerate(sizes):
        beams.append(_beam(int(n), intensity[b],
                           _coordinates(int(n), 1000 * (seed + 1) + b,
                                        case['form']), case['form']))
        maps.append(_transverse((chroma[b], chroma[b]), None) + [
            _longitudinal(True),
            _wakes(_bin_slicer(case['slices'], z_cuts=Z_CUTS), 1)])
    turn = BatchedTurn(BunchBatch(beams), maps)
    turn.track(6)
    return dict(kind='batch', turn=turn, form=case['form'])


def run(s):
    kind = s['kind']
    if kind == 'graph':
        s['turn'].replay(1)
        b = s['beam']
        # the last turn's kicks stay pending on xp and yp, as in the loop
        return {'x': b.x, 'y': b.y, 'z': b.z, 'dp': b.dp}
    if kind == 'batch':
        s['turn'].track(BATCH_TURNS)
        return dict(s['turn'].batch.storage, counts=s['turn'].counts)
    b = s['beam']
    if kind == 'slices':
        ss = s['slicer'].slice(b, statistics=list(SLICE_STATS))
        return dict({k: getattr(ss, k) for k in SLICE_STATS},
                    counts=ss.n_macroparticles_per_slice)
    for m in s['elements']:
        m.track(b)
    if kind == 'monitor':
        out = {k: getattr(b, k)() for k in BUNCH_STATS}
    else:
        ss = s['elements'][-1].slice_set_deque[0]
        out = {'counts': ss.n_macroparticles_per_slice, 'slice_x': ss.mean_x,
               'slice_y': ss.mean_y}
        if kind == 'eager':
            out.update(centroid_x=b.mean_x(), centroid_y=b.mean_y())
    if s['form'] == 'fp32':
        out = {k: float(v) for k, v in out.items()}
    out.update({k: getattr(b, k) for k in COORDS})
    return out


def work(case):
    """Bytes: every coordinate read and written once a turn (statistics:
    read once).  Operations: the maps' products and sums, a sine or cosine
    counted as ten."""
    size = 8 if case['form'] == 'fp64' else 4
    kind = case['kind']
    maps = 12 + 2 + 4     # transverse matrix, kicks, slice sums
    detuning = 30 + 4 * 10
    rf = 8 + 10
    if kind == 'graph':
        turns = max(1, case['wake_turns'])
        ops = maps + (detuning if case['detuned'] else 0) + \
            (rf if case['rf'] else 8)
        s, lags = case['slices'], case['wake_turns']
        wake = 2 * s * s * 2 * (1 + (lags if lags > 1 else 0))
        return {'bytes': turns * case['n'] * 12 * size,
                'flops': turns * (case['n'] * ops + wake)}
    if kind == 'batch':
        n = int(_batch_draws(case, 0)[0].sum()) * BATCH_TURNS
        return {'bytes': n * 12 * size, 'flops': n * (maps + 44 + rf)}
    if kind == 'slices':
        return {'bytes': case['n'] * 6 * size, 'flops': case['n'] * 44}
    n = case['n']
    if kind == 'monitor':
        ops = 12 + rf + 44 + (detuning if case['detuned'] else 0)
        return {'bytes': n * 18 * size, 'flops': n * ops}
    wake = case['slices']**2 * 2 * 4
    return {'bytes': n * 12 * size, 'flops': n * (maps + rf + 44) + wake}


# ------------------------------------------------- the same in 64 bits

BETA_REL = np.sqrt(1 - GAMMA**-2)
BETAGAMMA = np.sqrt(GAMMA**2 - 1)
P0 = BETAGAMMA * m_p * c


class _Bunch:
    def __init__(self, coords, intensity):
        for k, v in coords.items():
            setattr(self, k, v.double())
        self.per_mp = intensity / len(self.x)


def _map_transverse(b, chroma, amplitude):
    qx, qy = Q_X, Q_Y
    if chroma is not None:
        qx = qx + chroma[0] * b.dp
        qy = qy + chroma[1] * b.dp
    if amplitude is not None:
        jx = 0.5 * (b.x**2 / BETA + BETA * b.xp**2)
        jy = 0.5 * (b.y**2 / BETA + BETA * b.yp**2)
        qx = qx + (amplitude[0] * jx + amplitude[2] * jy) / P0
        qy = qy + (amplitude[1] * jy + amplitude[2] * jx) / P0
    for u, up, q in (('x', 'xp', qx), ('y', 'yp', qy)):
        phi = torch.as_tensor(q * (2 * np.pi), dtype=torch.float64,
                              device=b.x.device)
        cs, sn = torch.cos(phi), torch.sin(phi)
        v, vp = getattr(b, u), getattr(b, up)
        setattr(b, u, cs * v + BETA * sn * vp)
        setattr(b, up, -sn / BETA * v + cs * vp)


def _map_longitudinal(b, rf):
    eta = ALPHA_C - GAMMA**-2
    if rf:
        b.z = b.z - eta * b.dp * (0.5 * C_RING)
        amp = e * VOLTAGE / (BETA_REL * c)
        phi = HARMONIC * (2 * np.pi * b.z / C_RING)
        b.dp = (b.dp * P0 + amp * torch.sin(phi)) / P0
        b.z = b.z - eta * b.dp * (0.5 * C_RING)
        return
    omega_s = Q_S * (2 * np.pi * BETA_REL * c / C_RING)
    cs, sn = np.cos(2 * np.pi * Q_S), np.sin(2 * np.pi * Q_S)
    f = eta * BETA_REL * c / omega_s
    b.z, b.dp = b.z * cs - f * b.dp * sn, b.dp * cs + b.z / f * sn


def _resonator_wake(dt):
    r, freq, q = RESONATOR
    omega = 2 * np.pi * freq
    alpha = omega / (2 * q)
    bar = np.sqrt(np.abs(omega**2 - alpha**2))
    dt = dt.clip(max=0)
    return r * omega**2 / (q * bar) * np.exp(alpha * dt) * np.sin(bar * dt)


def _wall_wake(dt, yokoya=1.):
    radius, length, sigma, dt_min = WALL
    return (yokoya * (np.sign(dt + dt_min) - 1) / 2. * np.sqrt(BETA_REL) *
            length / np.pi / radius**3 *
            np.sqrt(-1. / np.pi / sigma / dt.clip(max=-dt_min)) *
            np.sqrt(119.9169832 * np.pi * c))


def _uniform_slices(b, n_slices, cuts):
    """Counts, sums of x and y per slice, the particles' slices (-1: out)."""
    tail, head = cuts
    width = (head - tail) / float(n_slices)
    idx = torch.floor((b.z - tail) / width).long()
    inside = (idx >= 0) & (idx < n_slices)
    return torch.where(inside, idx, torch.full_like(idx, -1))


def _per_slice(idx, n_slices, *values):
    """Counts and the sums of the values over the particles of each slice."""
    bins = idx + 1
    count = torch.bincount(bins, minlength=n_slices + 1)[1:n_slices + 1]
    return [count] + [torch.bincount(bins, weights=v, minlength=n_slices + 1)
                      [1:n_slices + 1] for v in values]


def _apply(b, target, idx, kick, factor=None):
    padded = torch.cat([torch.zeros(1, dtype=kick.dtype, device=kick.device),
                        kick])[idx + 1]
    setattr(b, target, getattr(b, target) +
            (padded if factor is None else padded * factor))


def _wake_factor(b):
    return -e**2 / (m_p * GAMMA * (BETA_REL * c)**2) * b.per_mp


class _Convolution:
    """The resonator and, over `turns` turns, the resistive wall on fixed
    or changing uniform cuts."""

    def __init__(self, n_slices, turns):
        self.n, self.turns = n_slices, turns
        self.past = []
        self.tables = {}

    def _toeplitz(self, cuts):
        if cuts not in self.tables:
            edges = cuts[0] + (cuts[1] - cuts[0]) / self.n * \
                np.arange(self.n + 1)
            t = (edges[:-1] + 0.5 * np.diff(edges)) / (BETA_REL * c)
            rows = []
            for lag in range(max(1, self.turns)):
                src = t + lag * C_RING / (BETA_REL * c)
                dt = np.concatenate((t - src[-1], (t - src[0])[1:]))
                w = _wall_wake(dt) if self.turns > 1 else 0 * dt
                rows.append(w + _resonator_wake(dt) if lag == 0 else w)
            self.tables = {cuts: torch.from_numpy(np.array(rows)).cuda()}
        return self.tables[cuts]

    def track(self, b, cuts):
        idx = _uniform_slices(b, self.n, cuts)
        count, sx, sy = _per_slice(idx, self.n, b.x, b.y)
        self.past = ([torch.stack([sx, sy])] + self.past)[:max(1, self.turns)]
        table = self._toeplitz(cuts)
        for k, target in enumerate(('xp', 'yp')):
            kick = 0
            for lag, m in enumerate(self.past):
                kick = kick + table[lag].unfold(0, self.n, 1) @ m[k].flip(0)
            _apply(b, target, idx, _wake_factor(b) * kick)
        return count, sx, sy


def _mean_or_zero(s, count):
    return torch.where(count > 0, s / count.clamp(min=1), 0 * s)


def _std(u):
    return torch.sqrt(((u - u.mean())**2).sum() / (len(u) - 1))


def _bunch_statistics(b):
    out = {'mean_' + k: getattr(b, k).mean() for k in COORDS}
    out.update({'sigma_' + k: _std(getattr(b, k))
                for k in ('x', 'y', 'z', 'dp')})
    dev = {k: getattr(b, k) - getattr(b, k).mean() for k in COORDS}

    def cov(p, q):
        return (dev[p] * dev[q]).sum() / (len(b.x) - 1)

    out.update(_emittances(cov, torch.sqrt))
    return {k: np.float64(float(out[k])) for k in BUNCH_STATS}


def _emittances(cov, sqrt):
    out = {}
    for u in 'xy':
        up = u + 'p'
        dd = cov('dp', 'dp')
        s11 = cov(u, u) - cov(u, 'dp')**2 / dd
        s12 = cov(u, up) - cov(u, 'dp') * cov(up, 'dp') / dd
        s22 = cov(up, up) - cov(up, 'dp')**2 / dd
        out['epsn_' + u] = sqrt(s11 * s22 - s12**2) * BETAGAMMA
    out['epsn_z'] = sqrt(cov('z', 'z') * cov('dp', 'dp') -
                         cov('z', 'dp')**2) * (4 * np.pi * P0 / e)
    return out


def _slice_statistics(b, case):
    n = case['slices']
    idx = _uniform_slices(b, n, SLICE_CUTS)
    count, *sums = _per_slice(idx, n, *[getattr(b, k) for k in COORDS])
    mean = {k: _mean_or_zero(s, count) for k, s in zip(COORDS, sums)}
    pad = {k: torch.cat([torch.zeros_like(m[:1]), m])[idx + 1]
           for k, m in mean.items()}
    dev = {k: getattr(b, k) - pad[k] for k in COORDS}

    def cov(p, q):
        return _per_slice(idx, n, dev[p] * dev[q])[1] / (count - 1)

    out = {'mean_' + k: mean[k] for k in COORDS}
    out.update({'sigma_' + k: torch.sqrt(cov(k, k))
                for k in ('x', 'y', 'z', 'dp')})
    out.update(_emittances(cov, torch.sqrt))
    return dict({k: out[k] for k in SLICE_STATS}, counts=count.int())


def _charge_turn(b, case, seed):
    n_slices, n = case['slices'], len(b.z)
    sz = float(_std(b.z))
    mz = float(b.z.mean())
    tail, head = mz - 3 * sz, mz + 3 * sz
    random.seed(int(seed))
    z, order = torch.sort(b.z)
    low = int((z < tail).sum())
    inside = n - low - int((z >= head).sum())
    extra = random.sample(list(range(n_slices)), inside % n_slices)
    per = (inside // n_slices) * np.ones(n_slices, dtype=int)
    per[extra] += 1
    first = low + np.concatenate([[0], np.cumsum(per)])
    idx = torch.full_like(order, -1)
    idx[order[low:low + inside]] = torch.from_numpy(
        np.repeat(np.arange(n_slices), per)).to(order.device)
    zh = z.cpu().numpy()
    edges = np.empty(n_slices + 1)
    edges[0], edges[-1] = tail, head
    edges[1:-1] = (zh[first[1:-1] - 1] + zh[first[1:-1]]) / 2
    t = (edges[:-1] + 0.5 * np.diff(edges)) / (BETA_REL * c)
    dt = t[None, :] - t[:, None]
    count, sx, sy = _per_slice(idx, n_slices, b.x, b.y)
    out = {'counts': count.int(), 'slice_x': sx / count, 'slice_y': sy / count}
    pi2 = np.pi**2
    f = _wake_factor(b)
    for target, moment, yokoya, quad in (
            ('xp', sx, pi2 / 24, None), ('xp', count.double(), -pi2 / 24, 'x'),
            ('yp', sy, pi2 / 12, None), ('yp', count.double(), pi2 / 24, 'y')):
        w = torch.from_numpy(_wall_wake(dt, yokoya)).to(moment.device)
        _apply(b, target, idx, f * (moment @ w),
               None if quad is None else getattr(b, quad))
    return out


def exact(case, seed):
    kind = case['kind']
    if kind == 'batch':
        return _exact_batch(case, seed)
    b = _Bunch(_coordinates(case['n'], seed, case['form']), INTENSITY)
    if kind == 'slices':
        return _slice_statistics(b, case)
    if kind == 'graph':
        chroma, amplitude = (CHROMA, AMPLITUDE) if case['detuned'] \
            else (None, None)
        wake = _Convolution(case['slices'], case['wake_turns'])
        for _ in range(_warmup(case) + case['wake_turns']):
            _map_transverse(b, chroma, amplitude)
            _map_longitudinal(b, case['rf'])
            wake.track(b, Z_CUTS)
        return {k: getattr(b, k) for k in ('x', 'y', 'z', 'dp')}
    if kind == 'monitor':
        chroma, amplitude = (CHROMA, AMPLITUDE) if case['detuned'] \
            else (None, None)
        _map_transverse(b, chroma, amplitude)
        _map_longitudinal(b, True)
        out = _bunch_statistics(b)
    elif kind == 'charge':
        _map_transverse(b, None, None)
        _map_longitudinal(b, True)
        out = _charge_turn(b, case, seed)
    else:
        _map_transverse(b, (2., 2.), None)
        _map_longitudinal(b, True)
        b.xp = b.xp - 2 / DAMPING * b.xp.mean()
        b.yp = b.yp - 2 / DAMPING * b.yp.mean()
        mz, sz = float(b.z.mean()), float(_std(b.z))
        count, sx, sy = _Convolution(case['slices'], 1).track(
            b, (mz - 3 * sz, mz + 3 * sz))
        # cuts that follow the bunch differ in the last bits of the mean:
        # a particle at an edge may count in either slice
        out = {'counts': None, 'slice_x': _mean_or_zero(sx, count),
               'slice_y': _mean_or_zero(sy, count),
               'centroid_x': np.float64(float(b.x.mean())),
               'centroid_y': np.float64(float(b.y.mean()))}
    out.update({k: getattr(b, k) for k in COORDS})
    return out


def _exact_batch(case, seed):
    sizes, chroma, intensity = _batch_draws(case, seed)
    pad = [-(-int(n) // 4) * 4 for n in sizes]
    out = {k: torch.zeros(sum(pad), dtype=torch.float64, device='cuda')
           for k in COORDS}
    counts = []
    at = 0
    for i, n in enumerate(sizes):
        b = _Bunch(_coordinates(int(n), 1000 * (seed + 1) + i, case['form']),
                   intensity[i])
        wake = _Convolution(case['slices'], 1)
        for turn in range(6 + BATCH_TURNS):
            _map_transverse(b, (chroma[i], chroma[i]), None)
            _map_longitudinal(b, True)
            # the last turn's kicks are still pending on the momenta
            xp, yp = b.xp, b.yp
            count, _, _ = wake.track(b, Z_CUTS)
        b.xp, b.yp = xp, yp
        counts.append(count.int())
        for k in COORDS:
            out[k][at:at + int(n)] = getattr(b, k)
        at += pad[i]
    # an FP32 particle at a slice edge may count in either slice
    return dict(out, counts=torch.stack(counts) if case['form'] == 'fp64'
                else None)
