"""The J/K build's chunking and scheduling: long contractions whose primitive
quartets are spread over lanes, every chunk order, builds in several threads.

Reference: the CPU oracle.  Tolerance 1e-10 on elements of order 1-10, the
parity bound of the FP64 kernels (sums of ~1e5 terms of 1e-16 relative
rounding each stay three orders below it)."""
import threading

import numpy
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.fixture(scope='module')
def b2():
    from pyscf_b200 import lib
    if lib.device_count() == 0:
        pytest.skip('no GPU')
    return lib


def contracted_molecule(nprims, l_of, ncopy=1, nctr=1):
    """atm, bas, env: one shell of nprims[k] primitives and angular momentum
    l_of[k] on its own atom, `ncopy` times over, about 1.5 Bohr apart."""
    rng = numpy.random.default_rng(42)
    env = [0.0] * 20
    atm, bas = [], []
    for c in range(ncopy):
        for k, (n, l) in enumerate(zip(nprims, l_of)):
            r = numpy.array([1.5 * k, 1.7 * c, 0.3 * (k + c)]) + rng.uniform(-0.1, 0.1, 3)
            atm.append([1, len(env), 1, len(env) + 3, 0, 0])
            env += list(r) + [0.0]
            e = 0.25 * 2.3 ** numpy.arange(n)
            bas.append([len(atm) - 1, l, n, nctr, 0, len(env), len(env) + n, 0])
            env += list(e) + list(rng.uniform(0.2, 1.0, n * nctr) / n)
    return (numpy.array(atm, dtype=numpy.int32), numpy.array(bas, dtype=numpy.int32), numpy.array(env))


def densities(nao, n):
    rng = numpy.random.default_rng(7)
    return rng.standard_normal((n, nao, nao)) / numpy.sqrt(nao)


# primitive pairs 1, 2, 4, 5, 16, 17, 81: both sides of every bucket's edge
@pytest.mark.parametrize('nprims,l_of,nctr', [
    ((1, 2, 4, 9), (0, 0, 0, 0), 1),
    ((1, 3, 5, 9), (1, 0, 1, 0), 1),
    ((2, 4, 1, 9), (2, 1, 0, 0), 1),
    ((4, 17, 1), (1, 0, 2), 2),
])
@pytest.mark.parametrize('hermi,n_dm', [(1, 1), (0, 2)])
def test_long_contractions(b2, nprims, l_of, nctr, hermi, n_dm):
    atm, bas, env = contracted_molecule(nprims, l_of, nctr=nctr)
    plan = b2.Plan(atm, bas, env, direct_scf_tol=1e-13)
    d = densities(plan.nao, n_dm)
    if hermi == 1:
        d = d + d.transpose(0, 2, 1)
    vj, vk = plan.get_jk(d, hermi=hermi)
    for s in range(n_dm):
        rj, rk, _ = oracle.get_jk(d[s], atm, bas, env, hermi=hermi)
        assert abs(vj[s] - rj).max() < TOL
        assert abs(vk[s] - rk).max() < TOL


@pytest.mark.parametrize('tile', [0, 1, 5, 64])
@pytest.mark.parametrize('tau', [0.0, 1e-3, 1e30])
def test_chunk_orders(b2, tile, tau):
    """Every tile size, with all quartets in float64, about half of them (by
    bound) or all in float32 (tau = 0, 1e-3, 1e30), J and K together and
    alone, against the oracle.  The float32 passes are held to 2e-5 of the
    largest element, as elsewhere."""
    atm, bas, env = contracted_molecule((1, 3, 9, 1), (1, 0, 0, 2), ncopy=6)
    plan = b2.Plan(atm, bas, env, direct_scf_tol=1e-13)
    d = densities(plan.nao, 1)[0]
    d = d + d.T
    rj, rk, _ = oracle.get_jk(d, atm, bas, env, hermi=1)
    plan.get_jk(d, hermi=1)
    nq = plan.stats()['quartets']
    plan.set_tile(tile)
    plan.set_mixed_threshold(tau)
    for kw in ({}, {'with_k': False}, {'with_j': False}):
        vj, vk = plan.get_jk(d, hermi=1, precision=b2.PREC_MIXED, **kw)
        st = plan.stats()
        assert st['quartets'] == nq
        assert (st['fp32_quartets'] == 0) if tau == 0.0 else (st['fp32_quartets'] == nq) if tau > 1.0 \
            else (nq // 4 < st['fp32_quartets'] < nq - nq // 4)
        for v, r in ((vj, rj), (vk, rk)):
            assert v is None or abs(v - r).max() < (TOL if tau == 0.0 else 2e-5 * abs(r).max())
        vj, vk = plan.get_jk(d, hermi=1, **kw)
        assert vj is None or abs(vj - rj).max() < TOL
        assert vk is None or abs(vk - rk).max() < TOL


def test_threads(b2):
    """Builds of different plans in several threads at once (each holds its
    own set of streams) give what they give alone."""
    atm, bas, env = contracted_molecule((1, 3, 9, 1), (1, 0, 0, 2), ncopy=3)
    plans = [b2.Plan(atm, bas, env, direct_scf_tol=1e-13) for _ in range(6)]
    d = densities(plans[0].nao, 6)
    want = [plans[0].get_jk(x + x.T, hermi=1) for x in d]
    bad = []

    def work(k):
        for _ in range(5):
            vj, vk = plans[k].get_jk(d[k] + d[k].T, hermi=1)
            if abs(vj - want[k][0]).max() > TOL or abs(vk - want[k][1]).max() > TOL:
                bad.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


@pytest.mark.parametrize('nprims,l_of,nctr', [
    ((1, 2, 4, 9), (0, 0, 0, 0), 1),
    ((1, 3, 5, 9), (1, 0, 1, 0), 1),
    ((2, 4, 1, 9), (2, 1, 0, 0), 1),
    ((4, 17, 1), (1, 0, 2), 2),
])
def test_long_contractions_gradient(b2, nprims, l_of, nctr):
    """The gradient J/K and the fused force of long contractions, whose
    primitive quartets are shared by lanes or lane groups."""
    atm, bas, env = contracted_molecule(nprims, l_of, nctr=nctr)
    plan = b2.Plan(atm, bas, env, direct_scf_tol=1e-13)
    d = densities(plan.nao, 1)[0]
    d = d + d.T
    rj, rk = oracle.grad_jk(d, atm, bas, env)[:2]
    vj, vk = plan.grad_jk(d)
    assert abs(vj - rj).max() < TOL
    assert abs(vk - rk).max() < TOL
    from pyscf_b200 import grad
    want = grad.grad_2e(rj, rk, d, grad.aoslice_by_atom(atm, bas))
    assert abs(plan.grad_contract(d) - want).max() < plan.nao * TOL


@pytest.mark.parametrize('nprims,l_of,nctr', [
    ((1, 2, 4, 9), (0, 0, 0, 0), 1),
    ((1, 3, 5, 9), (1, 0, 1, 0), 1),
    ((4, 17, 1), (1, 0, 2), 2),
])
def test_long_contractions_fill(b2, nprims, l_of, nctr):
    """The s8 tensor of long contractions (groups of a warp share a quartet's
    primitive quartets): J and K contracted from it on the host against the
    oracle's direct J and K."""
    atm, bas, env = contracted_molecule(nprims, l_of, nctr=nctr)
    plan = b2.Plan(atm, bas, env, direct_scf_tol=0.0)
    n = plan.nao
    eri = plan.int2e_s8(device=False)
    a = numpy.arange(n)
    hi, lo = numpy.maximum(a[:, None], a), numpy.minimum(a[:, None], a)
    tri = (hi * (hi + 1) // 2 + lo).ravel()
    p, q = numpy.maximum(tri[:, None], tri), numpy.minimum(tri[:, None], tri)
    full = eri[p * (p + 1) // 2 + q].reshape(n, n, n, n)
    d = densities(n, 1)[0]
    d = d + d.T
    rj, rk, _ = oracle.get_jk(d, atm, bas, env, hermi=1, screen=False)
    assert abs(numpy.einsum('ijkl,ji->kl', full, d) - rj).max() < TOL
    assert abs(numpy.einsum('ijkl,jk->il', full, d) - rk).max() < TOL


@pytest.mark.parametrize('nprims,l_of,ncopy', [
    ((1, 2, 3), (2, 1, 0), 5),      # (21|20), (21|11), (22|10): 5 groups of 6 lanes, 10 of 3
    ((1, 2), (3, 1), 4),            # (31|11), (31|31): 3 groups of 10 lanes
    ((1, 1, 2), (3, 2, 1), 2),      # (32|21), (32|11), (33|10): shares of the third index
])
@pytest.mark.parametrize('omega', [0.0, 0.4])
def test_row_family(b2, nprims, l_of, ncopy, omega):
    """The row family's classes on a chain whose distant kets fail the screen
    (survivors are compacted, the last round of groups is partly empty): one
    symmetric density, two general ones, J or K alone, the long-range operator,
    and every quartet in float32 (2e-5 of the largest element: the bound the
    float32 kernels are held to elsewhere)."""
    atm, bas, env = contracted_molecule(nprims, l_of, ncopy=ncopy)
    env[8] = omega
    for a in atm:
        env[a[1]] *= 3.0
        env[a[1] + 1] *= 2.5
    plan = b2.Plan(atm, bas, env, direct_scf_tol=1e-13)
    d = densities(plan.nao, 2)
    ds = d[0] + d[0].T
    rj, rk, _ = oracle.get_jk(ds, atm, bas, env, hermi=1)
    tol = TOL * max(1.0, abs(rj).max(), abs(rk).max())
    vj, vk = plan.get_jk(ds, hermi=1)
    assert abs(vj - rj).max() < tol and abs(vk - rk).max() < tol
    assert abs(plan.get_jk(ds, hermi=1, with_k=False)[0] - rj).max() < tol
    assert abs(plan.get_jk(ds, hermi=1, with_j=False)[1] - rk).max() < tol
    plan.set_mixed_threshold(1e30)
    fj, fk = plan.get_jk(ds, hermi=1, precision=b2.PREC_MIXED)
    assert abs(fj - rj).max() < 2e-5 * abs(rj).max() and abs(fk - rk).max() < 2e-5 * abs(rk).max()
    vj, vk = plan.get_jk(d, hermi=0)
    for s in range(2):
        rj, rk, _ = oracle.get_jk(d[s], atm, bas, env, hermi=0)
        assert abs(vj[s] - rj).max() < tol and abs(vk[s] - rk).max() < tol


def test_class_families(b2):
    """The class statistics tell the three kernel families apart: by the
    block's size, lanes (0), rows (2), and shared memory (1) for the six
    largest classes."""
    atm, bas, env = contracted_molecule((1, 1, 1, 1), (3, 2, 1, 0), ncopy=2)
    plan = b2.Plan(atm, bas, env, direct_scf_tol=1e-13)
    d = densities(plan.nao, 1)[0]
    plan.get_jk(d + d.T, hermi=1)
    fam = {(c['la'], c['lb'], c['lc'], c['ld']): c['family'] for c in plan.class_stats()}
    assert len(fam) == 55
    assert [fam[k] for k in ((0, 0, 0, 0), (1, 0, 0, 0), (2, 0, 1, 0), (3, 1, 0, 0))] == [0] * 4
    assert [fam[k] for k in ((1, 1, 1, 1), (2, 1, 2, 0), (2, 2, 2, 1), (3, 2, 2, 2))] == [2] * 4
    assert sorted(k for k in fam if fam[k] == 1) == [(3, 2, 3, 1), (3, 2, 3, 2), (3, 3, 2, 2), (3, 3, 3, 1),
                                                      (3, 3, 3, 2), (3, 3, 3, 3)]


def test_autotuner_leaves_rows(b2):
    """Variants 0 and 1 of a row class are the same launch: the autotuner does
    not choose between them."""
    atm, bas, env = contracted_molecule((1, 2, 1, 1), (2, 1, 0, 0), ncopy=4)
    plan = b2.Plan(atm, bas, env, direct_scf_tol=1e-13)
    d = densities(plan.nao, 1)[0]
    for _ in range(3):
        plan.autotune(d + d.T)
        for precision in (b2.PREC_FP64, b2.PREC_MIXED):
            rows = [v for v, c in zip(plan.tuning(precision), plan.class_stats()) if c['family'] == 2]
            assert len(rows) == 28 and not any(rows)


def test_classes_alone_and_side_by_side(b2):
    """A molecule of which some classes run alone, before the others run side
    by side, against all of them one after the other (class timing on): J/K,
    mixed, general densities, the gradient, the force, and in a batch with a
    small molecule.  The same sums in another order: 1e-12 of the largest."""
    import torch
    from conftest import load_fixture
    f, small = load_fixture('c20h42_vdz'), load_fixture('h2o_vdz')
    p = b2.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
    h = densities(p.nao, 1)[0]
    d, ds = torch.from_numpy(h).cuda(), torch.from_numpy(h + h.T).cuda()
    calls = [lambda: torch.stack(p.get_jk_device(ds, hermi=1)), lambda: torch.stack(p.get_jk_device(d, hermi=0)),
             lambda: torch.stack(p.grad_jk_device(ds)), lambda: p.grad_contract(ds)]
    for call in calls:
        p.set_profiling(True)
        want = call()
        nq = p.stats()['quartets'], p.grad_stats()['quartets']
        p.set_profiling(False)
        got = call()
        assert (p.stats()['quartets'], p.grad_stats()['quartets']) == nq
        assert float((got - want).abs().max()) < 1e-12 * max(1.0, float(want.abs().max()))
    q = b2.Plan(small['atm'], small['bas'], small['env'], direct_scf_tol=1e-13)
    e = densities(q.nao, 1)[0]
    e = torch.from_numpy(e + e.T).cuda()
    batch = b2.Batch([p, q])
    for precision in (b2.PREC_FP64, b2.PREC_MIXED):
        vj, vk = batch.get_jk_device([ds, e], hermi=1, precision=precision)
        for m, x, j, k in ((p, ds, vj[0], vk[0]), (q, e, vj[1], vk[1])):
            rj, rk = m.get_jk_device(x, hermi=1, precision=precision)
            for got, want in ((j, rj), (k, rk)):
                assert float((got - want).abs().max()) < 1e-12 * max(1.0, float(want.abs().max()))
