"""Fault handling on a GPU, without faulting the GPU.

* An out-of-memory condition is forced by the library's test hook
  (b200jk_debug_fail_alloc) instead of exhausting the device: plan creation
  and a build must return B200JK_ENOMEM, leave nothing behind, and the next
  calls must work.
* Host memory passed where device memory is declared is rejected on the host
  (cudaPointerGetAttributes) before any kernel could dereference it.
* A NaN density element propagates into J/K, as in the reference, and does
  not poison the plan for the next build.
"""
import ctypes

import numpy
import pytest

from conftest import load_fixture

pytestmark = pytest.mark.gpu

TOL_JK = 1e-10


@pytest.fixture(scope='module')
def b2():
    from pyscf_b200 import lib
    if lib.device_count() == 0:
        pytest.fail('no CUDA device visible to libb200jk')
    yield lib
    lib.load().b200jk_debug_fail_alloc(0)


@pytest.mark.parametrize('nth', [1, 3, 7])
def test_forced_enomem_in_plan_create(b2, nth):
    f = load_fixture('h2o_vdz')
    b2.load().b200jk_debug_fail_alloc(nth)
    try:
        with pytest.raises(b2.B200JKError) as e:
            b2.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
        assert e.value.code == b2.B200JK_ENOMEM
        assert 'cudaMalloc' in str(e.value)
    finally:
        b2.load().b200jk_debug_fail_alloc(0)
    p = b2.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
    vj, vk = p.get_jk(f['dm_rand'], hermi=1)
    assert abs(vj - f['vj_rand']).max() < TOL_JK
    assert abs(vk - f['vk_rand']).max() < TOL_JK


def test_forced_enomem_in_first_build(b2):
    """The first build allocates the workspace: a failure there is reported
    and the plan builds correctly on the next call."""
    f = load_fixture('h2o_vdz')
    p = b2.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
    b2.load().b200jk_debug_fail_alloc(2)
    try:
        with pytest.raises(b2.B200JKError) as e:
            p.get_jk(f['dm_rand'], hermi=1)
        assert e.value.code == b2.B200JK_ENOMEM
    finally:
        b2.load().b200jk_debug_fail_alloc(0)
    vj, vk = p.get_jk(f['dm_rand'], hermi=1)
    assert abs(vj - f['vj_rand']).max() < TOL_JK
    assert abs(vk - f['vk_rand']).max() < TOL_JK


def test_host_memory_as_device_pointers_rejected(b2):
    f = load_fixture('h2o_631g')
    p = b2.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
    dm = numpy.ascontiguousarray(f['dm_rand'])
    vj = numpy.empty_like(dm)
    vk = numpy.empty_like(dm)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    rc = b2.load().b200jk_get_jk(p._h, ptr(dm), 1, 1, 1, 1, ptr(vj), ptr(vk), 1, 0, None)
    assert rc == b2.B200JK_EINVAL
    rc = b2.load().b200jk_grad_jk(p._h, ptr(dm), 1, 1, 1, ptr(vj), ptr(vk), 1, 1e-14, None)
    assert rc == b2.B200JK_EINVAL
    # the same arrays as host arrays (dev_ptrs = 0) are fine
    vj2, vk2 = p.get_jk(dm, hermi=1)
    assert abs(vj2 - f['vj_rand']).max() < TOL_JK


def test_nan_density_propagates_and_plan_recovers(b2):
    f = load_fixture('h2o_vdz')
    p = b2.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
    dm = f['dm_rand'].copy()
    dm[0, 0] = float('nan')
    vj, vk = p.get_jk(dm, hermi=1)
    # J_ab = sum_cd (ab|cd) D_cd: every J element that meets D_00 is NaN, as
    # numpy would make it in the reference's driver
    assert numpy.isnan(vj).any()
    assert numpy.isnan(vj[0, 0]) and numpy.isnan(vk[0, 0])
    vj, vk = p.get_jk(f['dm_rand'], hermi=1)
    assert abs(vj - f['vj_rand']).max() < TOL_JK
    assert abs(vk - f['vk_rand']).max() < TOL_JK


@pytest.mark.parametrize('nth', [1, 2, 4])
def test_failed_gradient_replan_is_planned_again(b2, nth):
    """A tighter gradient tolerance whose longer pair lists cannot be
    allocated: the call at the first tolerance after it plans its lists again
    instead of using a mixture of the two."""
    f = load_fixture('h2o8_vdz')
    d = f['dm_rand'] + f['dm_rand'].T
    p = b2.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
    want = p.grad_jk(d, direct_scf_tol=1e-3)
    nq = p.grad_stats()['quartets']
    tight = b2.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13).grad_jk(d, direct_scf_tol=0.0)
    b2.load().b200jk_debug_fail_alloc(nth)
    try:
        with pytest.raises(b2.B200JKError) as e:
            p.grad_jk(d, direct_scf_tol=0.0)
        assert e.value.code == b2.B200JK_ENOMEM
    finally:
        b2.load().b200jk_debug_fail_alloc(0)
    for tol, ref in ((1e-3, want), (0.0, tight), (1e-3, want)):
        got = p.grad_jk(d, direct_scf_tol=tol)
        for g, r in zip(got, ref):
            assert abs(g - r).max() < TOL_JK * max(1.0, abs(r).max())
    assert p.grad_stats()['quartets'] == nq


def test_failed_item_list_of_the_stored_tensor(b2):
    """The stored-tensor contraction keeps the last basis size's item list per
    GPU: when the list of another size cannot be allocated, the next call at
    the first size makes its list again."""
    import torch
    from pyscf_b200 import incore
    rng = numpy.random.default_rng(3)
    cases = []
    for nao in (24, 9):
        npair = nao * (nao + 1) // 2
        eri = torch.from_numpy(rng.standard_normal(npair * (npair + 1) // 2)).cuda()
        d = rng.standard_normal((nao, nao))
        cases.append((eri, torch.from_numpy(d + d.T).cuda()))
    want = [torch.stack(incore.incore(e, d, hermi=1)) for e, d in reversed(cases)][::-1]
    incore.incore(*cases[0], hermi=1)      # the list of nao = 24 is there
    b2.load().b200jk_debug_fail_alloc(1)   # nao = 9 needs no larger workspace, only its list
    try:
        with pytest.raises(b2.B200JKError) as e:
            incore.incore(*cases[1], hermi=1)
        assert e.value.code == b2.B200JK_ENOMEM
    finally:
        b2.load().b200jk_debug_fail_alloc(0)
    for (eri, d), w in zip(cases, want):
        got = torch.stack(incore.incore(eri, d, hermi=1))
        assert float((got - w).abs().max()) < 1e-12 * float(w.abs().max())


def test_refused_allocation_does_not_fail_the_next_call(b2):
    """An allocation larger than the GPU (the s8 tensor of 760 functions, 335
    GB, into a host array that is never reached) is B200JK_ENOMEM, and the
    next build on another plan is not told of it."""
    import torch
    n = 760
    need = (n * (n + 1) // 2) * (n * (n + 1) // 2 + 1) // 2
    assert 8 * need > torch.cuda.get_device_properties(0).total_memory
    env = [0.0] * 20
    atm, bas = [], []
    for k in range(n):
        atm.append([1, len(env), 1, len(env) + 3, 0, 0])
        env += [20.0 * (k % 10), 20.0 * (k // 10 % 10), 20.0 * (k // 100), 0.0]
    for k in range(n):
        bas.append([k, 0, 1, 1, 0, len(env), len(env) + 1, 0])
    env += [1.0, 1.0]
    big = b2.Plan(numpy.array(atm, dtype=numpy.int32), numpy.array(bas, dtype=numpy.int32), numpy.array(env),
                  direct_scf_tol=1e-13)
    f = load_fixture('h2o_vdz')
    p = b2.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
    out = numpy.empty(1)
    rc = b2.load().b200jk_int2e_s8(big._h, out.ctypes.data_as(ctypes.c_void_p), need, 0, None)
    assert rc == b2.B200JK_ENOMEM
    vj, vk = p.get_jk(f['dm_rand'], hermi=1)
    assert abs(vj - f['vj_rand']).max() < TOL_JK
    assert abs(vk - f['vk_rand']).max() < TOL_JK
