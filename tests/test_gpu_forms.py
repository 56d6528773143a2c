"""The forms that the default dispatch chooses -- by batch size, contraction and output type -- against the CPU oracle,
at the sizes where one form hands over to the next.

ERI batches: the one-block sort ends at 4096 quartets; a long primitive loop is split over 2 to 16 lanes until the
batch is large (team kernels), or over 8, 4, 2 or 1 lanes by the quartet count ((xx|ss) kernels: on 148 SMs up to 9472,
25258 and 75776 quartets); a group may be partial.  The bound is the ERI bar, 1e-12 of the larger of one and the
batch's largest integral (sums of up to 625 terms of that size, each rounded a few times 1e-16); float output is the
FP64 value rounded once, 2^-24 of it, beside that bar.
J/K builds: uncontracted classes in groups, contracted ones in the list by primitive-loop length, both against the
oracle's direct build at the Fock bar, 1e-10.
"""
import numpy as np
import pytest

from qchem_b200 import api, basis as B, workloads as W

pytestmark = pytest.mark.gpu

ERI_ABS = 1e-12
FOCK_ABS = 1e-10


def _pool(npool, most, seed):
    """random shells like the benchmark's, contraction 1..most"""
    rng = np.random.default_rng(seed)
    return [B.Shell(L, tuple(rng.uniform(0.0, 6.0, size=3)), list(np.exp(rng.uniform(np.log(0.05), np.log(50.0), size=k))),
                    list(rng.uniform(0.1, 1.0, size=k)))
            for L in range(3) for k in rng.integers(1, most + 1, size=npool)]


@pytest.fixture(scope="module")
def engines(oracle_mod):
    made = {}

    def get(most):
        if most not in made:
            sh = _pool(96, most, 4700 + most)
            made[most] = (api.Engine(sh), oracle_mod.OracleBasis(sh))
        return made[most]
    return get


SMALL = [(0, 0, 0, 0), (2, 2, 0, 0), (1, 0, 1, 0), (2, 0, 1, 1), (2, 1, 2, 0), (2, 2, 2, 1)]


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("cls,most", [(c, m) for c in SMALL for m in (1, 3, 5) if m < 5 or sum(c) <= 4])
@pytest.mark.parametrize("nq", [1, 33, 257])
def test_small_batches(cls, nq, most, fp32, engines):
    """every quartet of small batches, whose loops are split over lanes; contraction 5 (up to 625 primitive quartets, in
    the light classes) goes beyond the pattern keys (4) and, for (xx|ss), beyond the ket pairs kept in shared memory"""
    eng, ob = engines(most)
    q = W.eri_class_batch(cls, nq, 96, seed=nq + most)
    got, ref = eng.eri_batch(cls, q, fp32=fp32), ob.eri_batch(q).reshape(nq, -1)
    assert got.dtype == (np.float32 if fp32 else np.float64)
    tol = ERI_ABS * max(1.0, np.abs(ref).max()) + (2.0 ** -24 * np.abs(ref) if fp32 else 0.0)
    assert np.all(np.abs(got.astype(np.float64) - ref) <= tol)


@pytest.mark.parametrize("cls,nq", [((0, 0, 0, 0), n) for n in (4096, 4097, 9472, 9473, 25258, 25259, 75777)]
                         + [((1, 1, 0, 0), 25259), ((2, 2, 0, 0), 9473), ((1, 0, 1, 0), 4096), ((1, 0, 1, 0), 4097),
                            ((1, 1, 1, 1), 20011), ((2, 1, 1, 0), 75777)])
def test_batches_at_the_edges_of_a_form(cls, nq, engines):
    eng, ob = engines(3)
    q = W.eri_class_batch(cls, nq, 96, seed=nq)
    pick = np.unique(np.concatenate([np.arange(200), np.arange(nq - 200, nq),
                                     np.random.default_rng(1).integers(0, nq, size=800)]))
    got = eng.eri_batch(cls, q)
    assert np.all(np.isfinite(got))
    ref = ob.eri_batch(q[pick]).reshape(len(pick), -1)
    assert np.abs(got[pick] - ref).max() <= ERI_ABS * max(1.0, np.abs(ref).max())


def test_fp32_batch_without_scratch_keeps_the_fp32_kernels(engines):
    """Under a memory limit that leaves no room for the team scratch the FP32 batch still runs (FP32 evaluation)."""
    cls, nq = (2, 2, 2, 2), 64
    sh = _pool(32, 3, 4750)
    q = W.eri_class_batch(cls, nq, 32, seed=5)
    free, tight = api.Engine(sh), api.Engine(sh)
    want = free.eri_batch(cls, q, fp32=True)
    tight.set_memory_limit(24 << 20)
    got = tight.eri_batch(cls, q, fp32=True)
    assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()


def _contracted(mol):
    """a split-valence contraction of the even-tempered exponents: contractions of 3, 2 and 1"""
    shells = []
    for sh in B.even_tempered(mol):
        k = round(np.log(sh.exps[0] / 0.1) / np.log(2.5))
        if shells and shells[-1].L == sh.L and shells[-1].atom == sh.atom and k >= 2 and len(shells[-1].exps) < 3 \
                and shells[-1].exps[0] > 0.5:
            shells[-1].exps.append(sh.exps[0])
            shells[-1].coefs.append(0.3)
        else:
            shells.append(B.Shell(sh.L, sh.centre, [sh.exps[0]], [1.0], sh.atom))
    return shells


def _density(n, seed=3):
    Q, _ = np.linalg.qr(np.random.default_rng(seed).normal(size=(n, 5)))
    return 2.0 * Q @ Q.T


@pytest.mark.parametrize("contracted", [False, True])
@pytest.mark.parametrize("waters", [1, 3])
def test_default_jk_matches_oracle(waters, contracted, oracle_mod):
    """The default forms: groups (one group to several per CTA), the list by loop length with split loops."""
    mol = W.water_cluster(nx=waters, ny=1, nz=1, seed=W.SEED0 + 3700)
    sh = _contracted(mol) if contracted else B.even_tempered(mol)
    assert not contracted or max(len(s.exps) for s in sh) == 3
    D = _density(B.nbf(sh))
    ob = oracle_mod.OracleBasis(sh)
    Jr, Kr = ob.jk_direct(D)[:2]
    eng = api.Engine(sh)
    J, K, _ = eng.fock_jk(D)
    assert np.abs(J - Jr).max() <= FOCK_ABS and np.abs(K - Kr).max() <= FOCK_ABS
    Jd, Kd, _ = eng.fock_jk(D, deterministic=True)
    assert np.abs(Jd - Jr).max() <= FOCK_ABS and np.abs(Kd - Kr).max() <= FOCK_ABS
    again = eng.fock_jk(D, deterministic=True)
    assert np.array_equal(Jd, again[0]) and np.array_equal(Kd, again[1])
    # a new threshold rebuilds the lists (the oracle screens alike: two thresholds differ by what they drop)
    eng.schwarz(1e-12)
    J2, K2, _ = eng.fock_jk(D)
    Jr, Kr = ob.jk_direct(D, thresh=1e-12)[:2]
    assert np.abs(J2 - Jr).max() <= FOCK_ABS and np.abs(K2 - Kr).max() <= FOCK_ABS


def test_contracted_jk_shards_batch_and_memory_limit():
    mol = W.water_cluster(nx=2, ny=1, nz=1, seed=W.SEED0 + 3710)
    sh = _contracted(mol)
    D = _density(B.nbf(sh))
    eng = api.Engine(sh)
    J, K, _ = eng.fock_jk(D)
    # shards take the work list as it is; their slices add up to the build
    Js, Ks = np.zeros_like(J), np.zeros_like(K)
    for r in range(3):
        eng.set_shard(r, 3)
        j, k, _ = eng.fock_jk(D)
        Js += j
        Ks += k
    assert np.abs(Js - J).max() <= FOCK_ABS and np.abs(Ks - K).max() <= FOCK_ABS
    # two molecules in one handle
    one, two = _contracted(W.water()), sh
    D1 = _density(B.nbf(one), seed=4)
    Jb, Kb, _ = api.BatchEngine([one, two]).fock_jk([D1, D])
    J1, K1, _ = api.Engine(one).fock_jk(D1)
    for x, y in ((Jb[0], J1), (Kb[0], K1), (Jb[1], J), (Kb[1], K)):
        assert np.abs(x - y).max() <= FOCK_ABS
    # without room for the scratch the thread-per-quartet form serves every class
    tight = api.Engine(sh)
    tight.schwarz()
    tight.set_memory_limit(8 << 20)
    Jt, Kt, _ = tight.fock_jk(D)
    assert np.abs(Jt - J).max() <= FOCK_ABS and np.abs(Kt - K).max() <= FOCK_ABS


@pytest.mark.parametrize("cls,most,nq", [((2, 1, 1, 0), 5, 3000), ((2, 2, 2, 2), 5, 220), ((1, 0, 1, 0), 8, 3000), ((2, 1, 2, 1), 6, 260)])
def test_long_loops_on_fewer_ctas(cls, most, nq, engines):
    """Contractions whose stage slots for a whole wave of CTAs would pass 4 GiB: as many CTAs as have room, each walking
    more groups; and counts of a few groups, which need few CTAs."""
    eng, ob = engines(most)
    q = W.eri_class_batch(cls, nq, 96, seed=nq + most)
    pick = np.random.default_rng(2).choice(nq, size=40, replace=False)
    ref = ob.eri_batch(q[pick]).reshape(len(pick), -1)
    for n in (nq, 63, 65):
        got = eng.eri_batch(cls, q[:n])
        use = pick < n
        assert np.abs(got[pick[use]] - ref[use]).max(initial=0.0) <= ERI_ABS * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("nq", [1, 31, 32, 33, 4097, 20001])
@pytest.mark.parametrize("cls", [(0, 0, 0, 0), (2, 2, 0, 0), (1, 0, 1, 0), (2, 1, 1, 1), (2, 2, 2, 2)])
def test_uncontracted_batches_are_not_sorted(cls, nq, fp32, oracle_mod, engines):
    """Batches of classes without contracted shells run in the order they come, up to partial groups and CTAs with
    several groups -- beside shells of another angular momentum that are contracted."""
    rng = np.random.default_rng(11)
    used = set(cls)
    sh = [B.Shell(L, tuple(rng.uniform(0.0, 6.0, size=3)), list(np.exp(rng.uniform(np.log(0.05), np.log(50.0), size=k))),
                  list(rng.uniform(0.1, 1.0, size=k)))
          for L in range(3) for k in ([1] * 40 if L in used else [3] * 40)]
    eng, ob = api.Engine(sh), oracle_mod.OracleBasis(sh)
    q = W.eri_class_batch(cls, nq, 40, seed=nq)
    pick = np.arange(nq) if nq < 100 else np.unique(np.concatenate([np.arange(40), np.arange(nq - 40, nq),
                                                                    rng.integers(0, nq, size=120)]))
    got, ref = eng.eri_batch(cls, q, fp32=fp32), ob.eri_batch(q[pick]).reshape(len(pick), -1)
    assert np.all(np.isfinite(got))
    tol = ERI_ABS * max(1.0, np.abs(ref).max()) + (2.0 ** -24 * np.abs(ref) if fp32 else 0.0)
    assert np.all(np.abs(got[pick].astype(np.float64) - ref) <= tol)
