"""The right-hand side of a periodic box on a uniform grid, in numpy, in any floating type: the
split-form sums of the framework's path from given fields (rho, u, v, w, T, p, H, mu)."""
import numpy as np


def _weights(n, T):
    q = lambda a, b: T(a) / T(b)  # noqa: E731
    return {1: ([0, q(1, 2)], [T(-2), T(1)]),
            2: ([0, q(2, 3), q(-1, 12)], [q(-5, 2), q(4, 3), q(-1, 12)]),
            3: ([0, q(3, 4), q(-3, 20), q(1, 60)], [q(-49, 18), q(3, 2), q(-3, 20), q(1, 90)]),
            4: ([0, q(4, 5), q(-1, 5), q(4, 105), q(-1, 280)],
                [q(-205, 72), q(8, 5), q(-1, 5), q(8, 315), q(-1, 560)])}[n]


def derived(p, f, T):
    """T, p, H, mu of the state f = (rho, u, v, w, rhoE), appended to rho, u, v, w."""
    r, u, v, w, e = (np.asarray(a).astype(T) for a in f)
    Rgas, gam = T(1.0 / ((p.gam * p.Ma) * p.Ma)), T(p.gam)
    t = (gam - 1) / Rgas * (e / r - (u * u + v * v + w * w) / 2)
    return [r, u, v, w, t, r * Rgas * t, e / r + Rgas * t, t ** T(p.viscexp) / T(p.Re)]


def rhs(p, f, T=np.longdouble):
    S, V = p.stencil_size, p.stencil_visc
    r, u, v, w, t, pr, h, m = derived(p, f, T)
    inv = [T(n) / T(L) for n, L in ((p.mx, p.Lx), (p.my, p.Ly), (p.mz, p.Lz))]
    c1S, (c1V, c2V) = _weights(S, T)[0], _weights(V, T)
    at = lambda a, d, l: np.roll(a, -l, axis=2 - d)  # noqa: E731
    d1 = lambda a, d, c: sum(c[k] * (at(a, d, k) - at(a, d, -k)) for k in range(1, len(c))) * inv[d]  # noqa: E731
    d2 = lambda a, d: (c2V[0] * a + sum(c2V[k] * (at(a, d, k) + at(a, d, -k))  # noqa: E731
                                        for k in range(1, V + 1))) * inv[d] ** 2
    U = [u, v, w]
    G = [[d1(U[c], d, c1V) for c in range(3)] for d in range(3)]
    th = G[0][0] + G[1][1] + G[2][2]
    acc, W, lap, cond, diss = [0 * r] * 5, [0 * r] * 3, [0 * r] * 4, 0 * r, 0 * r
    for d in range(3):
        for a in range(1, S + 1):
            c = c1S[a] * inv[d]
            qm = (at(r, d, -a) + r) * (at(U[d], d, -a) + U[d])
            qp = (at(r, d, a) + r) * (at(U[d], d, a) + U[d])
            acc[0] = acc[0] + c / 2 * (qm - qp)
            for n, E in enumerate((u, v, w, h), 1):
                acc[n] = acc[n] + c / 4 * (qm * at(E, d, -a) - qp * at(E, d, a))
        acc[1 + d] = acc[1 + d] - d1(pr, d, c1S)
        dm = d1(m, d, c1V)
        for c in range(3):
            tau = G[d][c] + G[c][d] - (T(2) / 3 * th if c == d else 0)
            W[c] = W[c] + tau * dm
            lap[c] = lap[c] + d2(U[c], d)
            diss = diss + tau * (G[2][1] if d == 1 and c == 2 and p.quirk_dissipation_y else G[d][c])
        W[d] = W[d] + m / 3 * d1(th, d, c1V)
        cond = cond + d1(t, d, c1V) * dm
        lap[3] = lap[3] + d2(t, d)
    for n, E in enumerate((u, v, w, h), 1):
        acc[n] = acc[n] + E * acc[0] / 2
    for c in range(3):
        W[c] = W[c] + m * lap[c]
        acc[1 + c] = acc[1 + c] + W[c]
    Ec = T(((p.gam - 1.0) * p.Ma) * p.Ma)
    acc[4] = acc[4] + m * diss + (cond + m * lap[3]) / (T(p.Pr) * Ec) + u * W[0] + v * W[1] + w * W[2]
    return acc
