"""Smearing, charge and reverse-mode differentiation in numpy, in whatever precision the fields have (64 or 80 bits):
quaternion fields of shape (4, T, X, Y, Z), each operation with its adjoint."""
import numpy as np


def qmul(a, b):
    a0, a1, a2, a3 = a
    b0, b1, b2, b3 = b
    return np.stack((a0 * b0 - a1 * b1 - a2 * b2 - a3 * b3, a0 * b1 + a1 * b0 - a2 * b3 + a3 * b2,
                     a0 * b2 + a1 * b3 + a2 * b0 - a3 * b1, a0 * b3 - a1 * b2 + a2 * b1 + a3 * b0))


def qdag(a):
    return np.stack((a[0], -a[1], -a[2], -a[3]))


class Node:
    """A value, what it was made from, and after backward() the gradient of the result with respect to it."""

    def __init__(self, value, parents=()):
        self.value, self.parents, self.grad = value, parents, None


def mul(a, b):
    return Node(qmul(a.value, b.value), ((a, lambda g: qmul(g, qdag(b.value))), (b, lambda g: qmul(qdag(a.value), g))))


def dag(a):
    return Node(qdag(a.value), ((a, qdag),))


def at(a, mu, k):
    """The field at x + k mu."""
    return Node(np.roll(a.value, -k, 1 + mu), ((a, lambda g: np.roll(g, k, 1 + mu)),))


def add(a, b):
    return Node(a.value + b.value, ((a, lambda g: g), (b, lambda g: g)))


def scale(a, c):
    return Node(a.value * c, ((a, lambda g: g * c),))


def unit(a):
    n = np.sqrt((a.value * a.value).sum(0))
    u = a.value / n
    return Node(u, ((a, lambda g: (g - u * (u * g).sum(0)) / n),))


def pure(a):
    def drop(x):
        return np.concatenate((np.zeros_like(x[:1]), x[1:]))
    return Node(drop(a.value), ((a, drop),))


def dot(a, b):
    return Node((a.value * b.value).sum(), ((a, lambda g: g * b.value), (b, lambda g: g * a.value)))


def backward(result):
    order, seen, stack = [], set(), [(result, 0)]
    while stack:
        x, i = stack.pop()
        if i == 0 and id(x) in seen:
            continue
        seen.add(id(x))
        if i < len(x.parents):
            stack += [(x, i + 1), (x.parents[i][0], 0)]
        else:
            order.append(x)
    result.grad = result.value.dtype.type(1)
    for x in reversed(order):
        for p, adjoint in x.parents:
            d = adjoint(x.grad)
            p.grad = d if p.grad is None else p.grad + d
        if x.parents:
            x.grad = None


def links(host, dims, dtype):
    """The four directions' links of a (V, 4, 4) array."""
    return [Node(np.ascontiguousarray(host[:, mu].T).reshape(4, *dims).astype(dtype)) for mu in range(4)]


def host(fields):
    return np.stack([f.reshape(4, -1).T for f in fields], 1)


def ape(U, mode, alpha):
    out = list(U)
    for mu in {"all": range(4), "spatial": range(1, 4), "temporal": range(1)}[mode]:
        nus = [nu for nu in range(4) if nu != mu and (mode == "all" or nu)]
        s = None
        for nu in nus:
            f = mul(mul(U[nu], at(U[mu], nu, 1)), dag(at(U[nu], mu, 1)))
            s = f if s is None else add(s, f)
        for nu in nus:
            b = at(U[nu], nu, -1)
            s = add(s, mul(mul(dag(b), at(U[mu], nu, -1)), at(b, mu, 1)))
        out[mu] = unit(add(U[mu], scale(s, alpha)))
    return out


def charge(U):
    num = U[0].value.dtype.type
    two = [mul(U[d], at(U[d], d, 1)) for d in range(4)]
    lines = {1: U, 2: two, 3: [mul(two[d], at(U[d], d, 2)) for d in range(4)]}

    def clover(A, B):
        total = None
        for e, k in ((1, num(3) / 2), (2, -num(3) / 20), (3, num(1) / 90)):
            a, b = lines[e][A], lines[e][B]
            ma, mb = at(a, A, -e), at(b, B, -e)
            leaves = (mul(mul(a, at(b, A, e)), mul(dag(at(a, B, e)), dag(b))),
                      mul(mul(dag(mb), at(a, B, -e)), mul(at(mb, A, e), dag(a))),
                      mul(mul(b, dag(at(ma, B, e))), mul(dag(at(b, A, -e)), ma)),
                      mul(mul(dag(ma), dag(at(mb, A, -e))), mul(at(ma, B, -e), mb)))
            for leaf in leaves:
                leaf = scale(leaf, k / 4)
                total = leaf if total is None else add(total, leaf)
        return pure(total)

    q = None
    for p, r in (((0, 1), (2, 3)), ((0, 2), (3, 1)), ((0, 3), (1, 2))):
        d = dot(clover(*p), clover(*r))
        q = d if q is None else add(q, d)
    pi = num("3.14159265358979323846264338327950288")
    return scale(q, -num(16) / (32 * pi * pi))


def charge_gradient(field, dims, n_ape, alpha, dtype):
    """dQ/dU as (V, 4, 3) su(2) coefficients."""
    U0 = links(field, dims, dtype)
    U = U0
    for _ in range(n_ape):
        U = ape(U, "all", dtype(alpha))
    backward(charge(U))
    return host([qmul(u.grad, qdag(u.value)) for u in U0])[:, :, 1:]


def smeared(field, dims, n, alpha, mode, dtype):
    U = links(field, dims, dtype)
    for _ in range(n):
        U = [Node(u.value) for u in ape(U, mode, dtype(alpha))]
    return host([u.value for u in U])
