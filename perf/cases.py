"""Performance cases of the RCWA raster path, each one pass through a public entry point.

Rasters are seeded binary stacks like the ones the workloads generate (rectangles and discs of
silicon-like permittivity in air, now and then a metal film), wavelengths 400-1600 nm on a 1 um cell,
oblique incidence. ``exact`` solves the same problems with LAPACK in 64 bits on the host.
"""
import math

import numpy as np
import torch

from wavebit_gb300 import adjoint, engine, rcwa

PERIOD = (1000.0, 1000.0)
EPS_TOP, EPS_BOT = 1.0, 2.25
LAYER_EPS = (2.25, 12.25)


def listed():
    return [
        # the documented first program: a 1D grating, one wavelength, the whole lifecycle in the default
        # (FP64) form; the smallest call a user makes, bound by launches and host work
        dict(name='grating_lifecycle', kind='lifecycle', hu=10, hv=0, L=1, B=1, ny=1, nx=4),
        # one small crossed grating, FP64: a convergence study's first steps
        dict(name='small_crossed_fp64', kind='solve', precision='double', hu=2, hv=2, L=1, B=1, ny=64, nx=64),
        # a ragged window, a few layers and points, FP64: a script's ordinary call
        dict(name='ragged_stack_fp64', kind='solve', precision='double', hu=4, hv=3, L=3, B=7, ny=96, nx=130),
        # an orders-(5,5) spectrum of a two-layer stack in the default form
        dict(name='crossed_spectrum_fp64', kind='solve', precision='double', hu=5, hv=5, L=2, B=16, ny=128, nx=128),
        # one request to an idle serving loop, mixed form: latency
        dict(name='request_mixed', kind='solve', precision='mixed', hu=5, hv=5, L=2, B=1, ny=128, nx=128),
        # the orders-(7,7) crossed-grating sweep in the mixed form, one matrix per SM
        dict(name='crossed_sweep_mixed', kind='solve', precision='mixed', hu=7, hv=7, L=4, B=32, ny=256, nx=256),
        # high orders, few points, mixed form: the largest window whose call stays within seconds
        dict(name='high_orders_mixed', kind='solve', precision='mixed', hu=10, hv=9, L=1, B=2, ny=256, nx=256),
        # stage A of a prepared stack: 256 x 256 rasters at the mixed sweep's orders
        dict(name='assemble_large', kind='assemble', hu=12, hv=12, L=4, B=1, ny=256, nx=256),
        # stage A of a small odd raster
        dict(name='assemble_small', kind='assemble', hu=5, hv=4, L=1, B=1, ny=101, nx=90),
        # stage C on kept modes (an eigenpair cache's hit): the FP64 cascade
        dict(name='cascade_fp64', kind='cascade', hu=7, hv=7, L=2, B=8, ny=128, nx=128),
        # the scattering matrix of a stack from kept modes (a stack cut in two and rejoined)
        dict(name='scattering_fp64', kind='scattering', hu=5, hv=5, L=2, B=4, ny=128, nx=128),
        # a gradient step of a patterned layer: forward and reverse through every stage
        dict(name='gradient_layer', kind='gradient', hu=5, hv=5, L=1, B=4, ny=128, nx=128),
    ]


def _odd(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))


def draw(rng):
    kind = rng.choice(['lifecycle', 'solve', 'solve', 'mixed', 'mixed', 'assemble', 'cascade', 'scattering',
                       'gradient'])
    ny, nx = _odd(rng, 40, 256), _odd(rng, 40, 256)
    if kind == 'lifecycle':
        return dict(kind=kind, hu=rng.randint(3, 30), hv=0, L=rng.randint(1, 3), B=rng.randint(1, 4), ny=1,
                    nx=rng.randint(4, 64))
    if kind == 'solve':
        return dict(kind='solve', precision='double', hu=rng.randint(1, 5), hv=rng.randint(1, 4), L=rng.randint(1, 3),
                    B=_odd(rng, 1, 24), ny=ny, nx=nx)
    if kind == 'mixed':
        return dict(kind='solve', precision='mixed', hu=rng.randint(2, 8), hv=rng.randint(2, 8), L=rng.randint(1, 4),
                    B=_odd(rng, 1, 32), ny=ny, nx=nx)
    if kind == 'assemble':
        return dict(kind=kind, hu=rng.randint(1, 12), hv=rng.randint(1, 12), L=rng.randint(1, 4), B=1, ny=ny, nx=nx)
    if kind == 'cascade':
        return dict(kind=kind, hu=rng.randint(2, 7), hv=rng.randint(2, 7), L=rng.randint(1, 3), B=_odd(rng, 1, 12),
                    ny=ny, nx=nx)
    if kind == 'scattering':
        return dict(kind=kind, hu=rng.randint(2, 5), hv=rng.randint(2, 5), L=rng.randint(1, 3), B=_odd(rng, 1, 6),
                    ny=ny, nx=nx)
    return dict(kind='gradient', hu=rng.randint(2, 5), hv=rng.randint(2, 4), L=rng.randint(1, 2), B=rng.randint(1, 5),
                ny=_odd(rng, 32, 128), nx=_odd(rng, 32, 128))


# ------------------------------------------------------------------------------- inputs
def _raster(rng, ny, nx):
    """Rectangles and discs of one material in air, about half the cell."""
    hi = LAYER_EPS[int(rng.integers(0, len(LAYER_EPS)))]
    a = np.ones((ny, nx), np.complex128)
    if ny == 1:
        edges = np.sort(rng.choice(np.arange(nx + 1), size=2, replace=False))
        a[0, edges[0]:edges[1]] = hi
        return a
    yy, xx = np.mgrid[0:ny, 0:nx]
    for _ in range(int(rng.integers(2, 5))):
        cy, cx = rng.uniform(0, ny), rng.uniform(0, nx)
        dy = np.abs((yy + 0.5 - cy + ny / 2) % ny - ny / 2) / ny
        dx = np.abs((xx + 0.5 - cx + nx / 2) % nx - nx / 2) / nx
        if rng.random() < 0.5:
            a[(dy < rng.uniform(0.08, 0.25)) & (dx < rng.uniform(0.08, 0.25))] = hi
        else:
            a[dy * dy + dx * dx < rng.uniform(0.1, 0.25) ** 2] = hi
    return a


def _problem(case, seed):
    rng = np.random.default_rng(seed)
    L, B = case['L'], case['B']
    eps = np.stack([_raster(rng, case['ny'], case['nx']) for _ in range(L)])
    if case['kind'] == 'solve' and L > 1:
        eps[L - 1, eps[L - 1] != 1.0] = -20 + 1.5j          # the last layer of a stack in metal
    p = dict(eps=eps, thick=rng.uniform(60., 300., size=L), wl=rng.uniform(500., 1500., size=B),
             theta=rng.uniform(0.05, 0.6, size=B), phi=rng.uniform(0.2, 1.3, size=B), pol=(0.6, 0.8))
    if case['kind'] == 'gradient':
        smooth = rng.standard_normal((L, case['ny'], case['nx']))
        f = np.exp(-0.5 * (np.fft.fftfreq(case['ny'])[:, None] ** 2 + np.fft.fftfreq(case['nx'])[None, :] ** 2)
                   * (2 * math.pi * 4.0) ** 2)
        smooth = np.fft.ifft2(np.fft.fft2(smooth) * f).real
        smooth /= smooth.std(axis=(1, 2), keepdims=True)
        p['eps'] = (1.0 + 11.25 / (1.0 + np.exp(-8.0 * smooth))).astype(np.complex128)
        p['theta'][:], p['phi'][:] = p['theta'][0], p['phi'][0]
        N = (2 * case['hu'] + 1) * (2 * case['hv'] + 1)
        p['wR'], p['wT'] = rng.uniform(0, 1, (B, N)), rng.uniform(0, 1, (B, N))
    if case['kind'] == 'lifecycle':
        p['theta'][:], p['phi'][:] = p['theta'][0], p['phi'][0]
        p['pol'] = (1.0, 0.0)
    return p


def _slots(eps, hu, hv):
    """Li's rule (fixed nesting, staircase series) of (ny, nx) in 64 bits: epx, epy, epz_i."""
    ny, nx = eps.shape
    dev = eps.device

    def series(npts, h):
        k = torch.arange(-2 * h, 2 * h + 1, dtype=torch.float64, device=dev)
        j = torch.arange(npts, dtype=torch.float64, device=dev)
        ph = torch.remainder(k[:, None] * j[None, :], npts) / npts
        t = k / npts
        return torch.exp(-2j * math.pi * ph) * (torch.sinc(t) * torch.exp(-1j * math.pi * t) / npts)[:, None]

    def toep(h):
        r = torch.arange(2 * h + 1, device=dev)
        return r[:, None] - r[None, :] + 2 * h

    nu, nv = 2 * hu + 1, 2 * hv + 1
    Fy, Fx, tu, tv = series(ny, hv), series(nx, hu), toep(hu), toep(hv)

    def nested(e):
        inner = torch.linalg.inv((Fy @ e).T[:, tv])                    # (nx, nv, nv)
        c = torch.einsum('kx,xrc->rck', Fx, inner)                     # (nv, nv, nku)
        return c[:, :, tu].permute(0, 2, 1, 3).reshape(nu * nv, nu * nv)

    direct = (Fy @ eps @ Fx.T)[tv][:, :, tu].permute(0, 2, 1, 3).reshape(nu * nv, nu * nv)
    return torch.linalg.inv(nested(eps)), nested(1.0 / eps), torch.linalg.inv(direct)


def _kxy(p, b, hu, hv, dev):
    u = torch.arange(-hu, hu + 1, dtype=torch.float64, device=dev) * (p['wl'][b] / PERIOD[0])
    v = torch.arange(-hv, hv + 1, dtype=torch.float64, device=dev) * (p['wl'][b] / PERIOD[1])
    s = math.sqrt(EPS_TOP) * math.sin(p['theta'][b])
    kx = (u[None, :] + s * math.cos(p['phi'][b])).expand(2 * hv + 1, -1).reshape(-1)
    ky = (v[:, None] + s * math.sin(p['phi'][b])).expand(-1, 2 * hu + 1).reshape(-1)
    return kx.contiguous(), ky.contiguous()


def _batch(p, case, dev='cuda'):
    L, B = case['L'], case['B']
    return engine.BatchInputs([list(range(L))] * B, [list(p['thick'])] * B, p['wl'], [PERIOD] * B, p['theta'],
                              p['phi'], [EPS_TOP] * B, [EPS_BOT] * B, [p['pol']] * B, device=dev)


def prepare(case, seed):
    p, hu, hv, kind = _problem(case, seed), case['hu'], case['hv'], case['kind']
    s = dict(kind=kind, hu=hu, hv=hv, precision=case.get('precision', 'double'))
    if kind == 'lifecycle':
        layers = tuple(rcwa.Layer(thickness=float(d), epsilon=e) for d, e in zip(p['thick'][::-1], p['eps'][::-1]))
        s['problem'] = rcwa.Problem(
            units=rcwa.Units('nm'),
            stack=rcwa.Stack(period=PERIOD, bottom=rcwa.Material(epsilon=EPS_BOT), layers=layers),
            excitation=rcwa.Excitation(wavelength=p['wl'],
                                       sources=(rcwa.PlaneWave(polarization='s', theta=float(p['theta'][0]),
                                                               phi=float(p['phi'][0])),)))
        s['numerics'] = rcwa.Numerics(orders=(hu, hv))
        return s
    s['eps'] = torch.as_tensor(p['eps'], device='cuda')
    if kind == 'assemble':
        return s
    if kind == 'gradient':
        s['p'] = p
        return s
    slots = [_slots(e, hu, hv) for e in s['eps']]
    s['conv'] = engine.ConvStack.from_matrices(*(torch.stack([t[k] for t in slots]) for k in range(3)), hu, hv)
    s['inp'] = _batch(p, case)
    if kind in ('cascade', 'scattering'):                    # the modes that such a program keeps
        k = [_kxy(p, b, hu, hv, 'cuda') for b in range(case['B']) for _ in range(case['L'])]
        _, q, W, V, _ = engine.layer_modes(s['conv'], np.tile(np.arange(case['L']), case['B']),
                                           torch.stack([a for a, _ in k]), torch.stack([a for _, a in k]),
                                           precision='mixed')
        s['modes'] = (W, V, q)
    return s


def run(s):
    kind, hu, hv = s['kind'], s['hu'], s['hv']
    if kind == 'lifecycle':
        r = rcwa.run(s['problem'], numerics=s['numerics'])
        return [r.R, r.T]
    if kind == 'solve':
        return list(engine.solve_batch(s['conv'], s['inp'], precision=s['precision']))
    if kind == 'assemble':
        c = engine.assemble(s['eps'], hu, hv)
        return [c.epx, c.epy, c.epz_i]
    if kind == 'cascade':
        return list(engine.smm_solve(*s['modes'], s['inp'], hu, hv, amplitudes=True))
    if kind == 'scattering':
        return list(engine.scattering_matrix(*s['modes'], s['inp'], hu, hv))
    p = s['p']
    return list(adjoint.solve_and_grad(s['eps'], p['thick'], p['wl'], PERIOD, hu, hv, p['wR'], p['wT'],
                                       theta=float(p['theta'][0]), phi=float(p['phi'][0]), eps_top=EPS_TOP,
                                       eps_bot=EPS_BOT, pol=p['pol'])[:5])


def work(case):
    """Real operations of the formulation: about 25 n^3 complex multiply-adds an eigen-solve, 53 n^3 flops a
    layer in the cascade; bytes: inputs and outputs once."""
    hu, hv, L, B = case['hu'], case['hv'], case['L'], case['B']
    N = (2 * hu + 1) * (2 * hv + 1)
    n = 2 * N
    raster, slots, modes = 16 * L * case['ny'] * case['nx'], 48 * L * N * N, 16 * B * L * (2 * n * n + n)
    stage_a = 8 * L * (2 * case['nx'] * (2 * hv + 1) * (case['ny'] + (2 * hv + 1) ** 2)
                       + 2 * (2 * hv + 1) ** 2 * (4 * hu + 1) * case['nx']) + 16 * L * N ** 3
    stage_b, stage_c = 200.0 * B * L * n ** 3, 53.0 * B * L * n ** 3
    kind = case['kind']
    if kind == 'assemble':
        return dict(bytes=raster + slots, flops=stage_a)
    if kind == 'cascade':
        return dict(bytes=modes + 48 * B * N, flops=stage_c)
    if kind == 'scattering':
        return dict(bytes=modes + 64 * B * n * n, flops=2 * stage_c + 96.0 * B * L * n ** 3)
    if kind == 'gradient':
        return dict(bytes=2 * raster + slots, flops=3 * stage_a + stage_b + 3 * stage_c + 100.0 * B * L * n ** 3)
    flops = stage_b + stage_c + (stage_a if kind == 'lifecycle' else 0)
    return dict(bytes=(raster if kind == 'lifecycle' else slots) + 48 * B * N, flops=flops)


# ------------------------------------------------------------------- the same in 64 bits
def _modes(kx, ky, epx, epy, epz):
    N = kx.numel()
    X, Y, eye = torch.diag(kx).to(epx.dtype), torch.diag(ky).to(epx.dtype), torch.eye(N, dtype=epx.dtype)
    left = torch.cat([torch.cat([X @ epz @ X - eye, X @ epz @ Y], 1), torch.cat([Y @ epz @ X, Y @ epz @ Y - eye], 1)])
    om2 = left @ torch.block_diag(epx, epy) + torch.cat([torch.cat([Y @ Y, -X @ Y], 1), torch.cat([-Y @ X, X @ X], 1)])
    omr = torch.cat([torch.cat([-X @ Y, X @ X - epy], 1), torch.cat([epx - Y @ Y, Y @ X], 1)])
    w, W = torch.linalg.eig(om2)
    q = torch.sqrt(w)
    q = torch.where(torch.where(q.real.abs() > 1e-12, q.real < 0, q.imag > 0), -q, q)
    return q, W, (omr @ W) / q


def _stack(p, b, hu, hv, slots, thick):
    """The half-spaces' waves and the layers' modes in the s/p basis of every order."""
    kx, ky = _kxy(p, b, hu, hv, 'cpu')
    kp2 = kx * kx + ky * ky
    kp = torch.sqrt(kp2)
    c, s = (kx / kp)[:, None], (ky / kp)[:, None]
    N, one = kx.numel(), torch.ones(kx.numel(), dtype=torch.complex128)
    kz = [torch.sqrt((e - kp2).to(torch.complex128)) for e in (EPS_TOP, EPS_BOT)]
    W0, V0 = zip(*((torch.cat([one, -1j * z / e]), torch.cat([-1j * z, one])) for z, e in zip(kz, (EPS_TOP, EPS_BOT))))
    layers = []
    for l in range(len(slots)):
        q, W, V = _modes(kx, ky, *slots[l])
        layers.append((torch.cat([c * W[N:] - s * W[:N], c * W[:N] + s * W[N:]]),
                       torch.cat([c * V[:N] + s * V[N:], c * V[N:] - s * V[:N]]),
                       torch.exp(-(2 * math.pi / p['wl'][b]) * thick[l] * q)))
    return kz, W0, V0, layers


def _reflect(W0, V0, layers, lit, far):
    """Reflection and transmission matrices of the stack lit from half-space ``lit``, in its port variables."""
    n = W0[0].numel()
    eye = torch.eye(n, dtype=torch.complex128)
    rho, steps = None, []
    E, H = torch.diag(W0[far]), torch.diag(V0[far])
    for W, V, X in layers[::-1] if lit == 0 else layers:
        P, Q = torch.linalg.solve(W, E), torch.linalg.solve(V, H)
        down = torch.linalg.inv(0.5 * (P + Q))
        rho = X[:, None] * (0.5 * (P - Q) @ down) * X
        steps.append(down * X)
        E, H = W @ (eye + rho), V @ (eye - rho)
    P, Q = E / W0[lit][:, None], H / V0[lit][:, None]
    down = torch.linalg.inv(0.5 * (P + Q))
    T = down
    for m in steps[::-1]:
        T = m @ T
    return 0.5 * (P - Q) @ down, T


def _efficiencies(kz, ref, trn, n_top, cols):
    N = kz[0].numel()
    spec = N // 2
    C = torch.zeros(2 * N, len(cols), dtype=torch.complex128)
    for j, (a, b) in enumerate(cols):
        C[spec, j], C[N + spec, j] = a, -1j * n_top * b
    r, t = ref @ C, trn @ C
    s0 = float(kz[0][spec].real)
    p0 = n_top ** 2 * float((kz[0][spec] / EPS_TOP).real)
    out, amps = [[], []], []
    for j, (a, b) in enumerate(cols):
        den = abs(a) ** 2 * s0 + abs(b) ** 2 * p0
        for k, (v, e) in enumerate(((r, EPS_TOP), (t, EPS_BOT))):
            z = kz[k]
            out[k].append((v[:N, j].abs() ** 2 * z.real + v[N:, j].abs() ** 2 * (z / e).real) / den)
        amps.append(torch.stack([r[:N, j], -r[N:, j] / (-1j * n_top), t[:N, j], t[N:, j] / (-1j * math.sqrt(EPS_BOT))]))
    return torch.stack(out[0]), torch.stack(out[1]), torch.stack(amps)


def exact(case, seed):
    hu, hv, L, B, kind = case['hu'], case['hv'], case['L'], case['B'], case['kind']
    N = (2 * hu + 1) * (2 * hv + 1)
    if kind not in ('assemble',) and B * L * (2 * N) ** 3 > 110 * 242 ** 3:
        return None                                          # LAPACK would take too long
    p = _problem(case, seed)
    grad = kind == 'gradient'
    eps = torch.tensor(p['eps'].real if grad else p['eps'], requires_grad=grad)
    thick = torch.tensor(p['thick'], requires_grad=grad)
    slots = [_slots(e.to(torch.complex128), hu, hv) for e in eps]
    if kind == 'assemble':
        return [torch.stack([t[k] for t in slots]) for k in range(3)]
    n_top = math.sqrt(EPS_TOP)
    cols = [p['pol'], (1.0, 0.0), (0.0, 1.0)]
    Rs, Ts, As, S = [], [], [], []
    sign = torch.tensor([(-1.0) ** (i % (2 * hu + 1) + i // (2 * hu + 1)) for i in range(N)] * 2)
    for b in range(B):
        kz, W0, V0, layers = _stack(p, b, hu, hv, slots, thick)
        ref, trn = _reflect(W0, V0, layers, 0, 1)
        if kind == 'scattering':
            # the mirrored stack: down-going columns of either orientation differ in the sign of H alone
            ref2, trn2 = _reflect(W0, V0, layers, 1, 0)
            S.append([sign[:, None] * m * sign for m in (ref, trn2, trn, ref2)])
            continue
        r, t, a = _efficiencies(kz, ref, trn, n_top, cols)
        Rs.append(r); Ts.append(t); As.append(a)
    if kind == 'scattering':
        return [torch.stack([m[k] for m in S]) for k in range(4)] + [None]
    if grad:
        R, T = torch.stack([r[0] for r in Rs]), torch.stack([t[0] for t in Ts])
        loss = (torch.tensor(p['wR']) * R).sum() + (torch.tensor(p['wT']) * T).sum()
        g_eps, g_th = torch.autograd.grad(loss, (eps, thick))
        return [loss.item(), R.detach(), T.detach(), g_eps, g_th]
    shape = (B, 3, 2 * hv + 1, 2 * hu + 1)
    R, T = torch.stack(Rs).reshape(shape), torch.stack(Ts).reshape(shape)
    if kind == 'lifecycle':
        return [R[:, 0], T[:, 0]]
    return [R, T, None] + ([torch.stack(As)] if kind == 'cascade' else [])
