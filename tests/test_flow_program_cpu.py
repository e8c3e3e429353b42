"""The task list of the dataflow factorisation / inverse, executed block by block in numpy in the order in which the
device takes it: every operand that a task reads must have been written by an earlier one (else a CTA could wait for
a task that nobody has taken), every tile is written once, and the result is the inverse or the Cholesky factor."""
import numpy as np
import pytest

from torchsso import _native as nat

T = 128
DIAG, PANEL, INVT, PROD = range(4)


def tasks_of(dims, with_inverse):
    lib = nat.lib()
    d = np.array(dims, dtype=np.int64)
    n = lib.sso_flow_tasks(len(dims), d.ctypes.data, with_inverse, None, 0)
    out = np.full((n, 4), -1, dtype=np.int16)
    assert lib.sso_flow_tasks(len(dims), d.ctypes.data, with_inverse, out.ctypes.data, n) == n
    return [tuple(int(v) for v in row) for row in out]


class Matrix:
    def __init__(self, m):
        self.m, self.np = m, (m.shape[0] + T - 1) // T
        self.W, self.X, self.Li, self.L, self.out = {}, {}, {}, {}, {}

    def block(self, i, j):
        return self.m[i * T:(i + 1) * T, j * T:(j + 1) * T]

    @staticmethod
    def put(tiles, key, value):
        assert key not in tiles, 'written twice'
        tiles[key] = value

    def run(self, kind, a, b, inverse):
        if kind == DIAG:
            assert a == b
            s = self.block(a, a) - sum(self.W[a, k] @ self.W[a, k].T for k in range(a))
            low = np.linalg.cholesky(s)
            self.put(self.L, a, low)
            self.put(self.Li, a, np.linalg.inv(low))
            if inverse:
                self.put(self.X, (a, a), self.Li[a].T)
        elif kind == PANEL:
            s = self.block(a, b) - sum(self.W[a, k] @ self.W[b, k].T for k in range(b))
            self.put(self.W, (a, b), s @ self.Li[b].T)
        elif kind == INVT:
            s = -sum(self.X[a, k] @ self.W[b, k].T for k in range(a, b))
            self.put(self.X, (a, b), s @ self.Li[b].T)
        else:
            t = sum(self.X[a, k] @ self.X[b, k].T for k in range(a, self.np))
            self.put(self.out, (a, b), t)
            if a != b:
                self.put(self.out, (b, a), t.T)


def matrices(dims):
    rng = np.random.default_rng(3)
    for d in dims:
        x = rng.standard_normal((2 * d + 8, d))
        yield Matrix(x.T @ x / x.shape[0] + 0.1 * np.eye(d))


DIMS = [[1], [128], [129, 5], [1000], [300, 1, 128, 577, 64, 384], [40] * 200 + [640, 641]]


@pytest.mark.parametrize('dims', DIMS)
@pytest.mark.parametrize('inverse', [True, False])
def test_tasks_in_their_order(dims, inverse):
    mats = list(matrices(dims))
    tasks = tasks_of(dims, int(inverse))
    assert len(set(tasks)) == len(tasks)
    for kind, mat, a, b in tasks:
        mats[mat].run(kind, a, b, inverse)      # a KeyError: an operand that no earlier task has written
    for m in mats:
        n = m.np
        if inverse:
            got = np.block([[m.out[i, j] for j in range(n)] for i in range(n)])
            assert np.allclose(got @ m.m, np.eye(len(m.m)), atol=1e-8)
        else:
            low = np.block([[m.L[i] if i == j else m.W.get((i, j), np.zeros((len(m.L[i]), len(m.L[j])))) for j in range(n)] for i in range(n)])
            assert np.allclose(low @ low.T, m.m, atol=1e-8)


def test_bad_arguments():
    lib = nat.lib()
    for dims in ([0], [-3], [1 << 20]):
        d = np.array(dims, dtype=np.int64)
        assert lib.sso_flow_tasks(1, d.ctypes.data, 1, None, 0) == -1
    assert lib.sso_flow_tasks(0, None, 1, None, 0) == -1
