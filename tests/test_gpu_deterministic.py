"""QCG_JK_DETERMINISTIC: the bits of a molecule's J and K depend on the molecule, its basis and the density only -- not
on how many quartets share the launches (groups per CTA, where primitive loops are cut), not on free memory."""
import numpy as np
import pytest

from qchem_b200 import api, basis as B, workloads as W
from tests.test_gpu_limits import _fill_device

pytestmark = pytest.mark.gpu

FOCK_ABS = 1e-10


def _contracted(mol, core):
    """contractions of `core`, three and one"""
    out = []
    for z, r in zip(mol.Z, mol.R):
        r = tuple(float(v) for v in r)
        for L, n in ((0, core), (0, 3), (0, 1), (1, 3), (1, 1), (2, 2)) if z == 8 else ((0, 3), (0, 1), (1, 1)):
            out.append(B.Shell(L, r, [0.25 * (n + L) * 2.7 ** k for k in range(n)][::-1], [0.4] * n))
    return out


def _density(n, seed=3):
    Q, _ = np.linalg.qr(np.random.default_rng(seed).normal(size=(n, 5)))
    return 2.0 * Q @ Q.T


def _shells(kind, mol):
    return B.even_tempered(mol) if kind == "even" else _contracted(mol, int(kind))


@pytest.mark.parametrize("kind", ["even", "3", "7"])
def test_alone_and_in_a_batch(kind, oracle_mod):
    mols = [W.water_cluster(nx=1, ny=1, nz=1, seed=W.SEED0 + 3800 + i) for i in range(64)]
    shells = [_shells(kind, m) for m in mols]
    Ds = [_density(B.nbf(sh), seed=i) for i, sh in enumerate(shells)]
    ref = {}
    for n in (1, 6, 64):
        J, K, _ = api.BatchEngine(shells[:n]).fock_jk(Ds[:n], deterministic=True)
        for i in range(min(n, 6)):
            if i not in ref:
                alone = api.Engine(shells[i]).fock_jk(Ds[i], deterministic=True)
                Jr, Kr = oracle_mod.OracleBasis(shells[i]).jk_direct(Ds[i])[:2]
                assert np.abs(alone[0] - Jr).max() <= FOCK_ABS and np.abs(alone[1] - Kr).max() <= FOCK_ABS
                ref[i] = alone
            assert np.array_equal(J[i], ref[i][0]) and np.array_equal(K[i], ref[i][1]), (n, i)


@pytest.mark.parametrize("kind", ["even", "3"])
def test_bits_do_not_depend_on_free_memory(kind):
    """No room for the scratch on the device: the default build takes another form, the deterministic one is refused,
    and with room again it gives the bits of any other handle."""
    import torch
    sh = _shells(kind, W.water_cluster(nx=2, ny=1, nz=1, seed=W.SEED0 + 3900))
    D = _density(B.nbf(sh))
    J, K, _ = api.Engine(sh).fock_jk(D, deterministic=True)
    eng = api.Engine(sh)
    eng.schwarz(1e-10)
    eng.set_memory_limit(1 << 20)   # the build's own buffers, no scratch
    eng.fock_jk(D)
    limited = eng.fock_jk(D, deterministic=True)   # under a limit: a form without scratch
    again = eng.fock_jk(D, deterministic=True)
    assert np.array_equal(limited[0], again[0]) and np.array_equal(limited[1], again[1])
    assert np.abs(limited[0] - J).max() <= FOCK_ABS and np.abs(limited[1] - K).max() <= FOCK_ABS
    eng.set_memory_limit(0)
    full = _fill_device()
    with pytest.raises(api.QcgError) as e:
        eng.fock_jk(D, deterministic=True)
    assert e.value.code == api.QCG_ERR_ALLOC
    Jt, Kt, _ = eng.fock_jk(D)
    assert np.abs(Jt - J).max() <= FOCK_ABS and np.abs(Kt - K).max() <= FOCK_ABS
    del full
    torch.cuda.empty_cache()
    Jd, Kd, _ = eng.fock_jk(D, deterministic=True)
    assert np.array_equal(Jd, J) and np.array_equal(Kd, K)
