"""Tables travel on the stream of the kernels that read them.

A plain cudaMemcpy from pageable memory may return before the data is on the
device and runs on the legacy stream, which the engine's non-blocking streams
do not wait for: a kernel launched next can read what the allocation held
before (on a new plan, an index out of any table).  The first test reads the
host sources for such copies; the others take the first gradient of many new
plans and moved geometries, whose bounds are computed from tables uploaded a
few microseconds earlier."""
import os
import re

import numpy
import pytest

from conftest import load_fixture

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'pyscf_b200', 'csrc')


def _statements(text):
    """The source without comments, cut into statements."""
    text = re.sub(r'/\*.*?\*/', '', re.sub(r'//[^\n]*', '', text), flags=re.S)
    return re.split(r'[;{}]', text)


def test_no_unordered_uploads():
    """Host-to-device copies and memsets name a stream; the copies to symbols
    (once per device) are followed by a wait."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(('.cu', '.cuh')):
            continue
        st = _statements(open(os.path.join(CSRC, name)).read())
        for i, s in enumerate(st):
            assert not re.search(r'\bcudaMemcpy\s*\(', s) or 'cudaMemcpyDeviceToHost' in s, s
            assert not re.search(r'\bcudaMemset\s*\(', s), s
            if re.search(r'\bcudaMemcpyToSymbol\s*\(', s):
                assert 'cudaStreamSynchronize' in s + st[i + 1], s


def _moved(f, seed):
    env = f['env'].copy()
    rng = numpy.random.default_rng(seed)
    for row in f['atm']:
        env[row[1]:row[1] + 3] += rng.uniform(-0.05, 0.05, 3)
    return env


@pytest.mark.gpu
@pytest.mark.parametrize('names,rounds', [(('h2o_631g', 'h2o_vdz'), 150), (('h2o_vdz', 'h2o8_vdz'), 25)])
def test_first_gradient_of_new_plans(names, rounds):
    """The derivative bounds of a new plan's first gradient J/K and first
    fused force are those of a plan that had the GPU to itself, whatever
    molecule the freed tables belonged to before.  Bounds: bitwise (maxima of
    sums in a fixed order); J/K and forces: 1e-10 (atomic sums)."""
    import torch
    from pyscf_b200 import lib
    if lib.device_count() == 0:
        pytest.skip('no GPU')
    fs = [load_fixture(n) for n in names]
    dms = [f['dm_rand'] + f['dm_rand'].T for f in fs]
    want = []
    for f, d in zip(fs, dms):
        torch.cuda.synchronize()
        p = lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
        torch.cuda.synchronize()
        q = p.grad_q_cond
        torch.cuda.synchronize()
        want.append((q, p.grad_jk(d), p.grad_contract(d)))
        p.close()
    for r in range(rounds):
        for f, d, (q, (vj, vk), de) in zip(fs, dms, want):
            p = lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
            if r % 2:
                assert abs(p.grad_contract(d) - de).max() < 1e-10 * max(1.0, abs(de).max())
            else:
                gj, gk = p.grad_jk(d)
                assert abs(gj - vj).max() < 1e-10 * max(1.0, abs(vj).max())
                assert abs(gk - vk).max() < 1e-10 * max(1.0, abs(vk).max())
            assert numpy.array_equal(p.grad_q_cond, q)
            p.close()


@pytest.mark.gpu
@pytest.mark.parametrize('name,rounds', [('h2o_vdz', 100), ('h2o8_vdz', 20)])
def test_first_gradient_of_moved_geometries(name, rounds):
    """One plan moved to and fro: bounds and forces of each geometry are those
    of a new plan there."""
    from pyscf_b200 import lib
    if lib.device_count() == 0:
        pytest.skip('no GPU')
    f = load_fixture(name)
    d = f['dm_rand'] + f['dm_rand'].T
    envs = [_moved(f, k) for k in range(3)]
    want = []
    for e in envs:
        p = lib.Plan(f['atm'], f['bas'], e, direct_scf_tol=1e-13)
        want.append((p.q_cond, p.grad_q_cond, p.grad_contract(d)))
        p.close()
    p = lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
    for r in range(rounds):
        k = r % 3
        p.update_coords(envs[k])
        de = p.grad_contract(d)
        assert abs(de - want[k][2]).max() < 1e-10 * max(1.0, abs(de).max())
        assert numpy.array_equal(p.q_cond, want[k][0])
        assert numpy.array_equal(p.grad_q_cond, want[k][1])


@pytest.mark.gpu
def test_tables_on_side_streams():
    """First calls on a caller's stream: the stored-tensor contraction's item
    list, the fill and the one-electron integrals are what the default stream
    gives."""
    import torch
    from pyscf_b200 import incore, lib
    if lib.device_count() == 0:
        pytest.skip('no GPU')
    f = load_fixture('h2o_vdz')
    d = torch.from_numpy(f['dm_rand'] + f['dm_rand'].T).cuda()
    ref = lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
    eri = ref.int2e_s8()
    S, H = ref.int1e(device=True)
    want = incore.incore(eri, d, hermi=1)
    small = torch.rand(21 * 22 // 2, dtype=torch.float64, device='cuda')
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(50):
            p = lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
            e = p.int2e_s8()
            s, h = p.int1e(device=True)
            incore.incore(small, torch.eye(6, dtype=torch.float64, device='cuda'), hermi=1)   # another item list
            vj, vk = incore.incore(e, d, hermi=1)
            side.synchronize()
            assert float((e - eri).abs().max()) < 1e-12
            assert torch.equal(s, S) and torch.equal(h, H)
            assert float((vj - want[0]).abs().max()) < 1e-10
            assert float((vk - want[1]).abs().max()) < 1e-10
            p.close()
