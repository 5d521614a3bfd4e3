"""Chains of 1-qubit channels applied in one pass (channel_1q_layer): the kernel on the CPU
emulator, and the library on the GPU, against the channels one by one in the oracle."""
import numpy as np
import pytest

import kemu
from oracle import restate as R
from test_emu_kernels import check_engine_counts, rand_rho

TOL = 1e-12


def rand_sop(rng):
    iso, _ = np.linalg.qr(rng.standard_normal((8, 2)) + 1j * rng.standard_normal((8, 2)))
    return R.kraus_to_superop([iso[2 * i:2 * i + 2] for i in range(4)])


# every mix of bits inside the sub-tile (below and above bit 3) and pairing bits; diagonal and
# off-diagonal items; blocks smaller than 64 x 64
@pytest.mark.parametrize("kind,lt", [("packed", 5), ("tiled", 5), ("tiled", 3)])
@pytest.mark.parametrize("n,qubits", [(2, (0, 1)), (3, (0, 2)), (5, (0, 1, 2, 3, 4)), (6, (0, 1, 2, 3, 4, 5)), (6, (1, 5)),
                                      (7, (0, 1, 2)), (7, (4, 5, 6)), (7, (0, 5, 6)), (7, (3, 4)), (7, (2, 6)), (8, (6, 7))])
def test_chain_emulated(kind, lt, n, qubits):
    rng = np.random.default_rng(sum(qubits) + n)
    rho = rand_rho(n, n)
    sops = [rand_sop(rng) for _ in qubits]
    if sum(q >= min(lt, 4) for q in qubits) > 2:               # more pairing bits than a block takes
        with pytest.raises(RuntimeError):
            kemu.dm_chain(kind, lt, R.to_storage(kind, rho, lt), n, qubits, sops)
        return
    res = kemu.dm_chain(kind, lt, R.to_storage(kind, rho, lt), n, qubits, sops)
    want = rho
    for q, s in zip(qubits, sops):
        want = R.apply_superop1(want, s, q)
    check_engine_counts(kind, n, lt, res)
    assert np.abs(res.out - R.to_storage(kind, want, lt)).max() < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("lt", [5, 3])
@pytest.mark.parametrize("kind", ["tiled", "packed"])
@pytest.mark.parametrize("n", [1, 2, 5, 6, 8, 9])
def test_layer_matches_oracle(kind, n, lt):
    """All qubits (chains of six, three and what is left), then a list with repeated qubits in
    falling order, whose channels do not commute."""
    import orkan_b200
    ork = orkan_b200.load(lt)
    rng = np.random.default_rng(n)
    rho = rand_rho(n, n + 1)
    for qubits in (list(range(n)), [q for q in reversed(range(n)) for _ in range(2)] + [0]):
        sops = np.stack([rand_sop(rng) for _ in qubits])
        st = ork.state(kind, n, R.to_storage(kind, rho, lt))
        ork.channel_1q_layer(st, sops, qubits)
        want = rho
        for q, s in zip(qubits, sops):
            want = R.apply_superop1(want, s, q)
        assert np.abs(ork.storage(st) - R.to_storage(kind, want, lt)).max() < TOL
        ork.free(st)
