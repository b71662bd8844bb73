"""The library's linear maps on uniform Cartesian levels of the unit cube in extended precision (numpy's long
double: 64 or 113 bits), and for each the sum of magnitudes that bounds an FP64 evaluation value by value."""
import numpy as np

LD = np.longdouble


def _legendre(m, z):
    p0, p1 = np.ones_like(z), z.copy()
    for j in range(2, m + 1):
        p0, p1 = p1, ((2 * j - 1) * z * p1 - (j - 1) * p0) / LD(j)
    return p1, m * (z * p1 - p0) / (z * z - 1)


def gauss(n):
    z = np.polynomial.legendre.leggauss(n)[0].astype(LD)
    for _ in range(3):
        p, d = _legendre(n, z)
        z = z - p / d
    d = _legendre(n, z)[1]
    return (1 + z) / 2, 1 / ((1 - z * z) * d * d)


def lobatto(n):
    if n == 2:
        return np.array([0, 1], LD)
    c = np.zeros(n)
    c[n - 1] = 1
    z = np.sort(np.real(np.polynomial.legendre.legroots(np.polynomial.legendre.legder(c)))).astype(LD)
    for _ in range(3):
        p, d = _legendre(n - 1, z)
        z = z - d * (1 - z * z) / (2 * z * d - (n - 1) * n * p)
    if n % 2:
        z[(n - 2) // 2] = 0
    return np.concatenate([[LD(0)], (1 + z) / 2, [LD(1)]])


def lagrange(z, x):
    """Values, first and second derivatives [basis, point] of the Lagrange basis on z."""
    n = len(z)
    V, D, E = (np.zeros((n, len(x)), LD) for _ in range(3))
    for i in range(n):
        f, f1, f2 = np.ones(len(x), LD), np.zeros(len(x), LD), np.zeros(len(x), LD)
        for j in range(n):
            if j != i:
                t = 1 / (z[i] - z[j])
                f2 = f2 * (x - z[j]) * t + 2 * f1 * t
                f1 = f1 * (x - z[j]) * t + f * t
                f = f * (x - z[j]) * t
        V[i], D[i], E[i] = f, f1, f2
    return V, D, E


def dg_1d(k, nc):
    """Mass and SIPG matrices of nc cells of degree k (FE_DGQ)."""
    n, h, gamma = k + 1, 1 / LD(nc), LD(k * (k + 1))
    z = lobatto(n)
    qx, qw = gauss(n)
    V, D, _ = lagrange(z, qx)
    G = lagrange(z, np.array([0, 1], LD))[1] / h
    M, A = np.zeros((nc * n, nc * n), LD), np.zeros((nc * n, nc * n), LD)
    for c in range(nc):
        s = slice(c * n, c * n + n)
        M[s, s] += (V * qw) @ V.T * h
        A[s, s] += (D * qw) @ D.T / h
    for f in range(nc + 1):
        jump, mean, inner = np.zeros(nc * n, LD), np.zeros(nc * n, LD), 0 < f < nc
        if f > 0:
            jump[f * n - 1] = 1
            mean[(f - 1) * n:f * n] = G[:, 1] * (LD(0.5) if inner else 1)
        if f < nc:
            jump[f * n] = -1
            mean[f * n:(f + 1) * n] += G[:, 0] * (LD(0.5) if inner else 1)
        i = slice(max(0, (f - 1) * n), min(nc, f + 1) * n)
        j, m = jump[i], mean[i]
        A[i, i] += gamma / h * (1 if inner else 2) * np.outer(j, j) - np.outer(m, j) - np.outer(j, m)
    return M, A


def embedding(k, nc):
    """FE_DGQ on nc cells to 2 nc cells."""
    n = k + 1
    z = lobatto(n)
    E = np.zeros((2 * nc * n, nc * n), LD)
    for s in range(2):
        V = lagrange(z, (z + s) / 2)[0]
        V[np.abs(V) < 1e-17] = 0
        for c in range(nc):
            E[(2 * c + s) * n:(2 * c + s + 1) * n, c * n:(c + 1) * n] = V.T
    return E


def q_1d(k, nc):
    """Mass, stiffness and C0IP bilaplacian of the interior nodes of nc cells (FE_Q)."""
    z, h, gamma = lobatto(k + 1), 1 / LD(nc), LD(k * (k + 1))
    qx, qw = gauss(k + 1)
    V, D, E = lagrange(z, qx)
    _, G, H = lagrange(z, np.array([0, 1], LD))
    n = nc * k + 1
    M, L, B = (np.zeros((n, n), LD) for _ in range(3))
    for c in range(nc):
        s = slice(c * k, c * k + k + 1)
        M[s, s] += (V * qw) @ V.T * h
        L[s, s] += (D * qw) @ D.T / h
        B[s, s] += (E * qw) @ E.T / h ** 3
    for f in range(nc + 1):
        jump, mean, inner = np.zeros(n, LD), np.zeros(n, LD), 0 < f < nc
        if f > 0:
            jump[(f - 1) * k:f * k + 1] += G[:, 1] / h
            mean[(f - 1) * k:f * k + 1] += H[:, 1] / h ** 2 * (LD(0.5) if inner else 1)
        if f < nc:
            jump[f * k:(f + 1) * k + 1] -= G[:, 0] / h
            mean[f * k:(f + 1) * k + 1] += H[:, 0] / h ** 2 * (LD(0.5) if inner else 1)
        i = slice(max(0, (f - 1) * k), min(n, (f + 1) * k + 1))
        j, m = jump[i], mean[i]
        B[i, i] += gamma / h * (1 if inner else 2) * np.outer(j, j) - np.outer(j, m) - np.outer(m, j)
    clean = lambda X: np.where(np.abs(X) < 1e-15 * np.abs(X).max(), LD(0), X)[1:-1, 1:-1]
    return clean(M), clean(L), clean(B)


def grid(u, nc, n):
    """Cell-wise numbering to the tensor over the 1-D indices (z, y, x)."""
    d = len(nc)
    g = np.asarray(u, LD).reshape(list(reversed(nc)) + [n] * d)
    return g.transpose([i for e in range(d) for i in (e, d + e)]).reshape([m * n for m in reversed(nc)])


def ungrid(g, nc, n):
    d = len(nc)
    g = g.reshape([m for c in reversed(nc) for m in (c, n)])
    return g.transpose([2 * e for e in range(d)] + [2 * e + 1 for e in range(d)]).reshape(-1)


def along(B, g, axis):
    """The banded matrix B along an axis."""
    o = np.zeros((B.shape[0],) + tuple(np.delete(g.shape, axis)), LD)
    g = np.moveaxis(g, axis, 0)
    for i in range(B.shape[0]):
        j = np.nonzero(B[i])[0]
        if j.size:
            o[i] = np.tensordot(B[i, j[0]:j[-1] + 1], g[j[0]:j[-1] + 1], axes=(0, 0))
    return np.moveaxis(o, 0, axis)


def _both(f, mats, x):
    return f(mats, x), f([[np.abs(B) for B in m] for m in mats], np.abs(x))


def sipg(k, nc, u):
    """SIPG operator times u, and the bound."""
    d = len(nc)

    def f(ops, g):
        out = np.zeros_like(g)
        for e in range(d):
            t = g
            for a in range(d):
                t = along(ops[a][1 if a == e else 0], t, d - 1 - a)
            out += t
        return out

    return [ungrid(v, nc, k + 1) for v in _both(f, [dg_1d(k, n) for n in nc], grid(u, nc, k + 1))]


def transfer(k, ncc, v, restrict):
    """Prolongation of a coarse vector or restriction of a fine one, and the bound."""
    d, nf = len(ncc), [2 * c for c in ncc]

    def f(ops, g):
        for a in range(d):
            g = along(ops[a][0], g, d - 1 - a)
        return g

    E = [embedding(k, c) for c in ncc]
    a, b = (nf, ncc) if restrict else (ncc, nf)
    return [ungrid(w, b, k + 1) for w in _both(f, [[e.T if restrict else e] for e in E], grid(v, a, k + 1))]


def c0ip(k, nc, x):
    """C0IP operator on nc x nc cells times x, and the bound."""
    n = nc * k - 1

    def f(ops, g):
        M, L, B = ops[0]
        return along(M, along(B, g, 1), 0) + 2 * along(L, along(L, g, 1), 0) + along(B, along(M, g, 1), 0)

    return [v.reshape(-1) for v in _both(f, [q_1d(k, nc)], np.asarray(x, LD).reshape(n, n))]


def smoother(k, nc, u, ncp):
    """Additive Schwarz sum of the patches' inverses of ncp cells per direction, and the bound |S| |1 / lambda| |S^T| |u| of its
    evaluation by fast diagonalization. The inverses come from that in FP64 and steps of iterative refinement."""
    d, n = len(nc), k + 1
    N, g = ncp * n, grid(u, nc, n)
    out, bound = np.zeros_like(g), np.zeros_like(g)

    def apply(mats, x):
        for e in range(d):
            x = np.moveaxis(np.tensordot(mats[e], x, axes=(1, d - 1 - e)), 0, d - 1 - e)
        return x

    patches = []
    for c in nc:
        M, A = dg_1d(k, c)
        patches.append([])
        for p in range(c - ncp + 1):
            s = slice(p * n, p * n + N)
            Li = np.linalg.inv(np.linalg.cholesky(M[s, s].astype(float)))
            lam, Q = np.linalg.eigh(Li @ A[s, s].astype(float) @ Li.T)
            patches[-1].append((M[s, s], A[s, s], Li.T @ Q, lam))
    for idx in np.ndindex(*[len(p) for p in patches]):
        P = [patches[e][idx[e]] for e in range(d)]
        at = tuple(slice(idx[e] * n, idx[e] * n + N) for e in reversed(range(d)))
        den = sum(P[e][3].reshape([-1 if d - 1 - e == a else 1 for a in range(d)]) for e in range(d))
        S = [p[2] for p in P]
        x, rest = np.zeros_like(g[at]), g[at]
        for _ in range(8):
            size = np.abs(rest).max()
            if size == 0:
                break
            x = x + size * apply(S, apply([s.T for s in S], (rest / size).astype(float)) / den)
            rest = g[at] - sum(apply([P[f][1] if f == e else P[f][0] for f in range(d)], x) for e in range(d))
        out[at] += x
        aS = [np.abs(s) for s in S]
        bound[at] += apply(aS, apply([s.T for s in aS], np.abs(g[at]).astype(float)) / den)
    return ungrid(out, nc, n), ungrid(bound, nc, n)


def worst(got, ref, bound):
    """Largest error over its bound, in units of 2^-53."""
    e = np.abs(np.asarray(got, LD) - ref)
    ok = bound > 0
    assert not np.any(e[~ok])
    return float((e[ok] / bound[ok]).max() * LD(2) ** 53)


def rms(got, ref):
    return float(np.sqrt(np.sum((np.asarray(got, LD) - ref) ** 2) / np.sum(ref ** 2)))


def spread(rows):
    """Largest row sum over the smallest entry that is not zero (up to rounding)."""
    a = np.abs(rows)
    return float(a.sum(1).max() / a[a > 1e-10 * a.max()].min())
