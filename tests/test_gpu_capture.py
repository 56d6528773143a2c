"""Device-pointer calls recorded into a caller's CUDA graph: buffers that the handle still has to allocate are allocated
during the capture, nothing that a replay would read elsewhere is uploaded in it, and replays follow their inputs."""
import ctypes

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


def _capture(stream, record):
    import torch
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        record()
    return graph


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("idle", [False, True])
def test_batches_of_new_classes(fp32, idle, oracle_mod):
    """Only one light class has run on the handle (its sort buffers are there, no scratch of the others is)."""
    import torch
    nq = 200
    classes = [(0, 0, 0, 0), (1, 0, 1, 0), (1, 1, 1, 0), (2, 0, 2, 0), (2, 2, 1, 1), (2, 2, 0, 0), (2, 2, 2, 2)]
    sh = _pool(32, 2, 4770)
    ob = oracle_mod.OracleBasis(sh)
    q = [torch.from_numpy(W.eri_class_batch(c, nq, 32, seed=k).astype(np.int32)).cuda() for k, c in enumerate(classes)]
    out = [torch.zeros(nq, int(np.prod([(l + 1) * (l + 2) // 2 for l in c])),
                       dtype=torch.float32 if fp32 else torch.float64, device="cuda") for c in classes]

    def batches(eng, which):
        for k in which:
            eng.eri_batch_device(classes[k], q[k].data_ptr(), nq, out[k].data_ptr(), fp32=fp32)

    api.lib().qcg_release_cache()
    if idle:
        other = api.Engine(sh)   # leaves scratch in the cache; its launches load the code as well
        batches(other, range(len(classes)))
        del other
    stream = torch.cuda.Stream()
    eng = api.Engine(sh)
    eng.set_stream(stream.cuda_stream)
    batches(eng, [0])
    torch.cuda.synchronize()
    graph = _capture(stream, lambda: batches(eng, range(1, len(classes))))
    for o in out:
        o.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    for k in range(1, len(classes)):
        ref = ob.eri_batch(q[k].cpu().numpy()).reshape(nq, -1)
        tol = ERI_ABS * max(1.0, np.abs(ref).max()) + (2.0 ** -24 * np.abs(ref) if fp32 else 0.0)
        assert np.all(np.abs(out[k].cpu().numpy().astype(np.float64) - ref) <= tol), classes[k]


@pytest.mark.parametrize("contracted", [False, True])
def test_first_build(contracted, oracle_mod):
    """A handle's first J/K build, with scratch of an earlier handle idle in the cache or not."""
    import torch
    mol = W.water()
    sh = B.even_tempered(mol)
    if contracted:
        sh = [B.Shell(x.L, x.centre, [x.exps[0], 2.7 * x.exps[0], 8.1 * x.exps[0]][:1 + i % 3], [1.0, 0.4, 0.2][:1 + i % 3])
              for i, x in enumerate(sh)]
    ob = oracle_mod.OracleBasis(sh)
    n = B.nbf(sh)
    D, J, K = (torch.zeros((n, n), dtype=torch.float64, device="cuda") for _ in range(3))
    f = api.lib().qcg_fock_jk_device
    for earlier in (False, True):
        if earlier:
            api.Engine(sh).fock_jk(np.eye(n))
        else:
            api.lib().qcg_release_cache()
        stream = torch.cuda.Stream()
        eng = api.Engine(sh)
        eng.set_stream(stream.cuda_stream)
        eng.schwarz(1e-10)
        args = [ctypes.c_void_p(x.data_ptr()) for x in (D, J, K)]
        flags = api.QCG_JK_SKIP_VALIDATION

        def record():
            assert f(eng._h, *args, flags, None) == api.QCG_OK, api.lib().qcg_last_error(eng._h).decode()

        graph = _capture(stream, record)
        eng.fock_jk(np.eye(n))   # goes on with the handle: its lists, its staging buffer
        eng.one_electron(mol)
        for seed in (1, 2):
            Q, _ = np.linalg.qr(np.random.default_rng(seed).normal(size=(n, 5)))
            D.copy_(torch.from_numpy(2.0 * Q @ Q.T))
            J.zero_(), K.zero_()
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            Jr, Kr = ob.jk_direct(D.cpu().numpy())[:2]
            assert np.abs(J.cpu().numpy() - Jr).max() <= FOCK_ABS and np.abs(K.cpu().numpy() - Kr).max() <= FOCK_ABS
