"""Batched solves over the ways a system is laid out: one CTA or a cluster of four, CG vectors
in registers, in shared memory or in the workspace, matrices that fit on chip and that do not.

Systems are random SPD matrices with a chain and long edges (so that a CTA's window of p is
narrow, or every column).  The residual is recomputed in numpy: with unit roundoff u and at
most W entries a row, the device's and numpy's FP64 residuals each carry an error of at most
(W + 2) u (|A| |x| + |b|), so the norm has to be <= rtol |b| + 2 (W + 2) u ||A| |x| + |b||.
A system's bits must not depend on the batch, nor on the order in which systems are taken.
"""

import numpy as np
import pytest
import scipy.sparse as sps
import torch

from tatva_gb300 import batched

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
RTOL = 1e-10


def _spd(n, extra, rng, shuffle):
    """Chain plus `extra` edges a row: neighbours within 40, or anywhere when shuffled."""
    i = np.arange(n - 1)
    rows, cols = [i], [i + 1]
    for _ in range(extra):
        a = np.arange(n)
        b = rng.integers(0, n, n) if shuffle else np.clip(a + rng.integers(2, 40, n), 0, n - 1)
        rows.append(a[a != b])
        cols.append(b[a != b])
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    w = rng.lognormal(0.0, 0.5, rows.size)
    S = sps.coo_matrix((w, (rows, cols)), shape=(n, n)).tocsr()
    S = S + S.T
    d = np.asarray(S.sum(axis=1)).ravel()
    return (sps.diags(1.02 * d + 1e-3) - S).tocsr()


def _systems(mats, dev):
    A = sps.block_diag(mats, format="csr")
    A.sort_indices()
    ofs = np.concatenate([[0], np.cumsum([m.shape[0] for m in mats])])
    t = lambda a, d: torch.from_numpy(a.astype(d)).to(dev)  # noqa: E731
    return batched.BatchedSystems(t(A.indptr, np.int32), t(A.indices, np.int32),
                                  t(A.data, np.float64), ofs)


# (rows, extra edges a row, numbering shuffled)
KINDS = [
    (1, 0, False), (2, 0, False), (33, 1, False), (511, 2, True),   # one CTA
    (2300, 1, False),            # one CTA; more rows than registers hold at 512 threads
    (2561, 1, False),            # smallest cluster by rows: 641, 641, 641, 638
    (2601, 2, True),             # cluster, every window holds all of p
    (700, 20, True),             # cluster by the width of the rows
    (2401, 30, False),           # the matrix does not fit: part of each row in global memory
    (9409, 2, False), (10240, 1, True),   # largest with vectors in registers (256 threads)
    (10243, 1, False),           # vectors in shared memory
    (45001, 1, True),            # p takes the SM: vectors in the workspace
]


@pytest.mark.parametrize("threads", [128, 256, 512])
def test_every_layout_reaches_the_residual(cuda, threads):
    rng = np.random.default_rng(5)
    mats = [_spd(n, e, rng, s) for n, e, s in KINDS]
    bs = [rng.standard_normal(m.shape[0]) for m in mats]
    sysm = _systems(mats, cuda)
    b = torch.from_numpy(np.concatenate(bs)).to(cuda)
    res = sysm.solve(b, rtol=RTOL, threads=threads)
    assert res.converged, res.status
    xs = [x.cpu().numpy() for x in sysm.split(res.x)]
    for kind, m, bb, x in zip(KINDS, mats, bs, xs):
        W = int(np.diff(m.indptr).max())
        err = np.linalg.norm(bb - m @ x)
        bound = RTOL * np.linalg.norm(bb) + 2 * (W + 2) * U * np.linalg.norm(
            abs(m) @ np.abs(x) + np.abs(bb))
        assert err <= bound, (kind, err / np.linalg.norm(bb))
    # the other way round (small systems first, clusters and single CTAs interleaved)
    sysm.order_d.copy_(sysm.order_d.flip(0))
    assert torch.equal(sysm.solve(b, rtol=RTOL, threads=threads).x, res.x)
    for k in (3, 5, 8, 10):
        alone = _systems([mats[k]], cuda)
        x1 = alone.solve(torch.from_numpy(bs[k]).to(cuda), rtol=RTOL, threads=threads).x
        assert np.array_equal(x1.cpu().numpy(), xs[k]), KINDS[k]


@pytest.mark.parametrize("threads,n", [(128, 511), (128, 513), (256, 1024), (256, 1025)])
def test_many_small_systems(cuda, threads, n):
    """Enough systems for the launch with more CTAs on an SM (and one row too many for it):
    same bits as alone."""
    rng = np.random.default_rng(7)
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    mats = [_spd(int(k), 1, rng, False) for k in rng.integers(3, 60, 8 * sms)] + \
        [_spd(n, 1, rng, False)]
    bs = [rng.standard_normal(m.shape[0]) for m in mats]
    sysm = _systems(mats, cuda)
    res = sysm.solve(torch.from_numpy(np.concatenate(bs)).to(cuda), rtol=RTOL, threads=threads)
    assert res.converged
    xs = sysm.split(res.x)
    for k in (0, 100, len(mats) - 1):
        alone = _systems([mats[k]], cuda)
        x1 = alone.solve(torch.from_numpy(bs[k]).to(cuda), rtol=RTOL, threads=threads).x
        assert torch.equal(x1, xs[k])


def test_breakdown_in_a_cluster(cuda):
    """A non-positive diagonal entry anywhere in a large system is reported, and the other
    systems of the batch are solved."""
    rng = np.random.default_rng(9)
    good, bad = _spd(3000, 1, rng, False), _spd(5000, 1, rng, False).tolil()
    bad[4999, 4999] = -1.0
    sysm = _systems([good, bad.tocsr(), good], cuda)
    b = torch.ones(11000, dtype=torch.float64, device=cuda)
    res = sysm.solve(b)
    assert list(res.status) == [0, 7, 0] and res.rel_res[1] == 1.0
    xs = sysm.split(res.x)
    assert torch.equal(xs[0], xs[2])
