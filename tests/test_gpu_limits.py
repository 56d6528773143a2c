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


@pytest.mark.parametrize("idle", [0, 4800])
def test_scratch_stays_within_the_limit(idle):
    """A batch whose scratch is just above a power of two, and one that could take a larger idle buffer: what the
    handle holds is within its limit (beside the slabs of 8 MiB that small buffers share)."""
    import torch
    sh = _pool(16, 1, 4760)
    cls, nq, limit = (2, 2, 2, 2), 120, 88 << 20

    def batch(eng, n):
        q = torch.from_numpy(W.eri_class_batch(cls, n, 16, seed=1).astype(np.int32)).cuda()
        out = torch.empty(n, 1296, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        eng.eri_batch_device(cls, q.data_ptr(), n, out.data_ptr())
        torch.cuda.synchronize()
        return out.cpu().numpy()

    want = batch(api.Engine(sh), nq)
    api.lib().qcg_release_cache()
    eng = api.Engine(sh)
    if idle:
        batch(api.Engine(sh), idle)   # leaves its scratch, several times larger, in the cache
    eng.set_memory_limit(limit)
    assert np.array_equal(batch(eng, nq), want)
    # with the cache's idle buffers freed, what the handle's end gives back is what it held
    api.lib().qcg_release_cache()
    before = torch.cuda.mem_get_info()[0]
    del eng
    api.lib().qcg_release_cache()
    assert torch.cuda.mem_get_info()[0] - before <= limit + (16 << 20)


def test_optional_scratch_makes_room(oracle_mod):
    """What fits a limit by itself still fits after calls whose fastest form keeps scratch: batches and J/K builds in
    turn, under limits from just their own buffers up to all the scratch."""
    sh = [x for x in _contracted(W.water()) if len(x.exps) <= 3]
    ob = oracle_mod.OracleBasis(sh)
    D = _density(B.nbf(sh))
    Jr, Kr = ob.jk_direct(D)[:2]
    s, p = ([i for i, x in enumerate(sh) if x.L == L] for L in (0, 1))
    rng = np.random.default_rng(2)
    nq = 20
    q = np.stack([rng.choice(p, nq), rng.choice(s, nq), rng.choice(p, nq), rng.choice(s, nq)], axis=1).astype(np.int32)
    ref = ob.eri_batch(q).reshape(nq, -1)

    def jk(eng):
        J, K, _ = eng.fock_jk(D)
        assert np.abs(J - Jr).max() <= FOCK_ABS and np.abs(K - Kr).max() <= FOCK_ABS

    def batch(eng):
        got = eng.eri_batch((1, 0, 1, 0), q, fp32=True)
        assert np.abs(got - ref).max() <= 2e-5 * max(1.0, np.abs(ref).max())

    def least(call):
        lo, hi = 1, 1 << 26
        while hi - lo > 64:
            mid = (lo + hi) // 2
            eng = api.Engine(sh)
            eng.schwarz(1e-10)
            eng.set_memory_limit(mid)
            try:
                call(eng)
                hi = mid
            except api.QcgError as e:
                assert e.code == api.QCG_ERR_ALLOC
                lo = mid
        return hi

    # what the screening and each call's own buffers take (a subset mask of at most 256 bytes measures the former)
    assert len(sh) ** 2 <= 256
    screening = least(lambda eng: eng.set_pair_subset(np.ones((len(sh), len(sh)), dtype=np.uint8))) - 256
    both = least(jk) + least(batch) - screening + 256
    for order in ((jk, batch), (batch, jk)):
        for extra in range(0, 24 << 20, 96 << 10):
            eng = api.Engine(sh)
            eng.schwarz(1e-10)
            eng.set_memory_limit(both + extra)
            for call in order + order:
                call(eng)


def test_idle_scratch_gives_way_to_other_allocations():
    """With the device full but for less than the next call needs, the idle scratch of an earlier handle goes: a batch
    with large host buffers and a network's activations both find room."""
    import torch
    sh = [B.Shell(2, (0.1 * i, 0.0, 0.3 * i), [0.3, 1.1, 4.0], [0.3, 0.5, 0.4]) for i in range(8)]
    q = np.random.default_rng(0).integers(0, 8, size=(60000, 4)).astype(np.int32)   # 622 MB of integrals
    want = api.Engine(sh).eri_batch((2, 2, 2, 2), q)   # the same batch: a smaller one may split its primitive loops
    rows = 50000
    x, y = torch.randn(rows, 29, device="cuda"), torch.empty(rows, 1225, device="cuda")
    net = api.Mlp([29, 64, 1225])
    net.forward(64, x.data_ptr(), y.data_ptr())
    torch.cuda.synchronize()

    def fill():
        """idle scratch of 512 MiB and more, and the rest of the device taken but for about 400 MiB"""
        eng = api.Engine(sh)
        eng.eri_batch((2, 2, 2, 2), q[:20000])
        del eng
        torch.cuda.synchronize()
        return torch.empty(torch.cuda.mem_get_info()[0] - (400 << 20), dtype=torch.uint8, device="cuda")

    full = fill()
    net.forward(rows, x.data_ptr(), y.data_ptr())   # four arrays of 245 MB
    torch.cuda.synchronize()
    del full, net
    torch.cuda.empty_cache()
    assert torch.isfinite(y).all().item()
    eng = api.Engine(sh)
    eng.eri_batch((2, 2, 2, 2), q[:20000])   # keeps its scratch, and buffers of 207 MB that the next call outgrows
    full = fill()
    got = eng.eri_batch((2, 2, 2, 2), q)
    assert np.array_equal(got, want)
    del full
    torch.cuda.empty_cache()


def _fill_device():
    """every piece of device memory down to 2 MiB; the tensors that hold it"""
    import torch
    api.lib().qcg_release_cache()
    torch.cuda.empty_cache()
    full, size = [], torch.cuda.mem_get_info()[0]
    while size >= 2 << 20:
        try:
            full.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            size //= 2
    return full


def test_calls_after_scratch_found_no_room(oracle_mod):
    """A float batch and a J/K build on a full device, more than once, run in forms without scratch, a double batch is
    refused each time; with room again all of them are right."""
    import torch
    sh = B.even_tempered(W.water_cluster(nx=2, ny=1, nz=1, seed=W.SEED0 + 3740))
    ob = oracle_mod.OracleBasis(sh)
    D = _density(B.nbf(sh))
    Jr, Kr = ob.jk_direct(D)[:2]
    d = [i for i, x in enumerate(sh) if x.L == 2]
    q = np.random.default_rng(0).choice(d, size=(400, 4)).astype(np.int32)
    ref = ob.eri_batch(q).reshape(400, -1)
    eng = api.Engine(sh)
    eng.schwarz(1e-10)

    def float_batch():
        assert np.abs(eng.eri_batch((2, 2, 2, 2), q, fp32=True) - ref).max() <= 2e-5 * max(1.0, np.abs(ref).max())

    def build():
        J, K, _ = eng.fock_jk(D)
        assert np.abs(J - Jr).max() <= FOCK_ABS and np.abs(K - Kr).max() <= FOCK_ABS

    # the calls' own buffers, and the code of the forms without scratch; host buffers of the double batch too
    eng.eri_batch((2, 2, 0, 0), np.repeat(np.array([[d[0], d[0], 0, 0]], dtype=np.int32), 15000, axis=0))
    small = api.Engine(sh)
    small.schwarz(1e-10)
    small.set_memory_limit(6 << 20)
    small.fock_jk(D)
    small.eri_batch((2, 2, 2, 2), q[:100], fp32=True)
    full = _fill_device()
    for _ in range(3):
        float_batch()
        build()
        _refused(lambda: eng.eri_batch((2, 2, 2, 2), q))
    del full
    torch.cuda.empty_cache()
    for _ in range(2):
        float_batch()
        build()
        assert np.abs(eng.eri_batch((2, 2, 2, 2), q) - ref).max() <= ERI_ABS * max(1.0, np.abs(ref).max())
