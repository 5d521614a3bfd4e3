"""Diagonal gates on packed density matrices of more than 10 qubits, column by column in storage order
(orkan_b200/csrc/cuda/dm_phase.cuh), and the pass by items beside it: the lowest and highest qubits and those
between, lines of half a block, one and two of them, one, two and three qubits, against the elementwise definition, on the emulator with every
access counted and on the GPU."""
import numpy as np
import pytest

import kemu
from oracle import restate as R

TOL = 1e-14
CASES = [("z", (0,)), ("t", (4,)), ("sdg", (9,)), ("p", (10,)), ("rz", (3,)), ("rz", (-1,)), ("cz", (0, 10)),
         ("cz", (-1, 9)), ("cz", (1, 2))]


def phases(name, n, qs, th):
    psi = np.ones(1 << n, complex)
    return R.apply_pure(psi, name, qs, th)


def random_storage(n, seed):
    rng = np.random.default_rng(seed)
    d = 1 << n
    size = d * (d + 1) // 2
    return rng.standard_normal(size) + 1j * rng.standard_normal(size)


def expected(st, n, ph):
    d = 1 << n
    out, o = st.copy(), 0
    for c in range(d):
        out[o:o + d - c] *= ph[c:] * np.conj(ph[c])
        o += d - c
    return out


def cases(n):
    for name, qs in CASES:
        qs = tuple(q % n for q in qs)
        yield name, qs, 0.7 if name in ("p", "rz") else None


def test_emulated():
    n = 11
    st = random_storage(n, 1)
    for name, qs, th in cases(n):
        k = len(qs)
        small = R.apply_pure(np.ones(1 << k, complex), name, tuple(range(k))[::-1], th)
        res = kemu.dm_phase("packed", 5, st, n, list(qs), small)
        assert res.oob == 0
        assert res.reads.max() == 1 and (res.reads == res.writes).all()
        want = expected(st, n, phases(name, n, qs, th))
        assert np.abs(res.out - want).max() <= TOL * np.abs(st).max()
    three = np.exp(1j * np.arange(8))
    res = kemu.dm_phase("packed", 5, st, n, [10, 0, 4], three)
    x = np.arange(1 << n)
    local = (x >> 10 & 1) << 2 | (x & 1) << 1 | (x >> 4 & 1)
    assert res.oob == 0 and (res.reads == res.writes).all()
    assert np.abs(res.out - expected(st, n, three[local])).max() <= TOL * np.abs(st).max()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [11, 12, 13])
def test_on_the_gpu(ork5, n):
    host = random_storage(n, n)
    for name, qs, th in cases(n):
        st = ork5.state("packed", n)
        ork5.upload(st, host)
        ork5.gate(st, name, qs, th)
        got = ork5.storage(st)
        ork5.free(st)
        assert np.abs(got - expected(host, n, phases(name, n, qs, th))).max() <= TOL * np.abs(host).max()
