"""Handles that cannot have all the device memory they ask for: a call that fails leaves the handle usable, a form that
is chosen for speed makes room for what a call cannot do without, and the cap on a handle's memory is kept."""
import numpy as np
import pytest

from qchem_b200 import api, basis as B, workloads as W

pytestmark = pytest.mark.gpu

FOCK_ABS = 1e-10
ERI_ABS = 1e-12


def _pool(n, most, seed):
    rng = np.random.default_rng(seed)
    return [B.Shell(L, tuple(rng.uniform(0.0, 6.0, size=3)), list(np.exp(rng.uniform(np.log(0.05), np.log(50.0), size=k))),
                    list(rng.uniform(0.1, 1.0, size=k)))
            for L in range(3) for k in rng.integers(1, most + 1, size=n)]


def _density(n, seed=3):
    Q, _ = np.linalg.qr(np.random.default_rng(seed).normal(size=(n, 5)))
    return 2.0 * Q @ Q.T


def _refused(call):
    with pytest.raises(api.QcgError) as e:
        call()
    assert e.value.code == api.QCG_ERR_ALLOC


def test_buffers_that_could_not_grow(oracle_mod):
    """A batch, and a J/K build, that find no room leave no address of released memory: what the handle allocates next
    and a smaller batch after it do not meet."""
    sh = B.even_tempered(W.water())
    eng, ob = api.Engine(sh), oracle_mod.OracleBasis(sh)
    cls = (1, 0, 0, 0)
    s, p = ([i for i, x in enumerate(sh) if x.L == L] for L in (0, 1))
    q = np.array([[p[i % len(p)], s[i % 3], s[i % 5], s[i % 2]] for i in range(300)], dtype=np.int32)
    ref = ob.eri_batch(q).reshape(300, -1)
    assert np.abs(eng.eri_batch(cls, q[:60]) - ref[:60]).max() <= ERI_ABS
    eng.set_memory_limit(1)
    _refused(lambda: eng.eri_batch(cls, q))
    eng.set_memory_limit(0)
    eng.schwarz(1e-10)
    eng.set_memory_limit(1)
    D = _density(eng.nbf)
    _refused(lambda: eng.fock_jk(D))
    eng.set_memory_limit(0)
    Jr, Kr = ob.jk_direct(D)[:2]
    for n in (60, 20, 300):
        J, K, _ = eng.fock_jk(D)
        assert np.abs(J - Jr).max() <= FOCK_ABS and np.abs(K - Kr).max() <= FOCK_ABS
        assert np.abs(eng.eri_batch(cls, q[:n]) - ref[:n]).max() <= ERI_ABS


def _contracted(mol):
    """contractions of six, three and one: the primitive loops of a class have many lengths"""
    out = []
    for z, r in zip(mol.Z, mol.R):
        r = tuple(float(v) for v in r)
        for L, n in ((0, 6), (0, 3), (0, 1), (1, 3), (1, 1)) if z == 8 else ((0, 3), (0, 1), (1, 1)):
            out.append(B.Shell(L, r, [0.25 * (n + L) * 2.7 ** k for k in range(n)][::-1], [0.4] * n))
    return out


def test_builds_under_a_limit_that_holds_part_of_a_list(oracle_mod):
    """The contracted form's lists (three arrays a class) under every limit between none of them and all: many builds
    in a row give the same J and K, and none takes memory that the next one misses."""
    sh = _contracted(W.water_cluster(nx=2, ny=1, nz=1, seed=W.SEED0 + 3720))
    D = _density(B.nbf(sh))
    Jr, Kr = oracle_mod.OracleBasis(sh).jk_direct(D)[:2]

    def screened():
        eng = api.Engine(sh)
        eng.schwarz(1e-10)
        return eng

    def fits(limit, builds):
        eng = screened()
        eng.set_memory_limit(limit)
        try:
            for _ in range(builds):
                J, K, _ = eng.fock_jk(D)
                assert np.abs(J - Jr).max() <= FOCK_ABS and np.abs(K - Kr).max() <= FOCK_ABS
        except api.QcgError as e:
            assert e.code == api.QCG_ERR_ALLOC
            return False
        return True

    lo, hi = 1, 1 << 26   # one build fits in hi and not in lo
    assert fits(hi, 1) and not fits(lo, 1)
    while hi - lo > 256:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if fits(mid, 1) else (mid, hi)
    # what the lists take is of the order of the work lists: 256 bytes and more per array
    for extra in (0, 256, 512, 1024, 2048, 4096, 8192, 16384, 32768, 65536, 1 << 17):
        eng = screened()
        eng.set_memory_limit(hi + extra)
        for _ in range(30):
            J, K, _ = eng.fock_jk(D)
            assert np.abs(J - Jr).max() <= FOCK_ABS and np.abs(K - Kr).max() <= FOCK_ABS
        # the room beyond the build's own buffers is still there: a new subset mask (one byte a shell pair, 484)
        if extra >= 512:
            eng.set_pair_subset(np.ones((len(sh), len(sh)), dtype=np.uint8))
