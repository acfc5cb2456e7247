"""The stream sets builds run on: every allocation, stream creation and lane of
a first J/K, gradient and fill made to fail in turn.  Each failure is an error
code, nothing is left running, and the next call on the same plan is right."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.join(os.path.dirname(os.path.abspath(__file__)), '..')

# In a process of its own: sets are kept while a device has plans, so only
# the first build after the last plan has gone creates one.
SCRIPT = r'''
import sys
sys.path[:0] = ['.', 'tests']
import numpy
from conftest import load_fixture
from pyscf_b200 import lib
f = load_fixture('h2o_631g')
d = f['dm_rand'] + f['dm_rand'].T
calls = {
    'jk': lambda p: numpy.array(p.get_jk(d, hermi=1)),
    'grad': lambda p: numpy.array(p.grad_jk(d)),
    'force': lambda p: p.grad_contract(d),
    'fill': lambda p: p.int2e_s8(device=False),
}
call = calls[sys.argv[1]]
new = lambda: lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
p = new()
want = call(p)
p.close()
streams = nth = 0
while True:
    nth += 1
    p = new()
    lib.load().b200jk_debug_fail_alloc(nth)
    try:
        got = call(p)
        failed = False
    except lib.B200JKError as e:
        failed = True
        assert e.code in (lib.B200JK_ENOMEM, lib.B200JK_ECUDA), e
        assert (e.code == lib.B200JK_ECUDA) == ('(test hook)' in str(e)), e
        streams += 'stream creation' in str(e)
    lib.load().b200jk_debug_fail_alloc(0)
    got = call(p)
    assert abs(got - want).max() < 1e-10 * max(1.0, abs(want).max()), nth
    p.close()
    if not failed:
        break
assert nth < 200 and streams == 7, (nth, streams)
print('ok', nth)
'''


@pytest.mark.parametrize('call', ['jk', 'grad', 'force', 'fill'])
def test_failing_stream_sets(call):
    r = subprocess.run([sys.executable, '-c', SCRIPT, call], cwd=ROOT, stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.startswith(b'ok'), r.stdout.decode()[-2000:]


@pytest.mark.parametrize('op', ['jk', 'grad', 'fill', 'batch'])
@pytest.mark.parametrize('nth', [2, 8, 17])
def test_error_between_fork_and_join_waits(op, nth):
    """A launch that fails with others in flight: the call returns once those
    have ended (the caller's stream is idle), and the next call is right."""
    import torch
    from conftest import load_fixture
    from pyscf_b200 import lib
    if lib.device_count() == 0:
        pytest.skip('no GPU')
    f = load_fixture('h2o8_vdz')
    d = torch.from_numpy(f['dm_rand'] + f['dm_rand'].T).cuda()
    plans = [lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13) for _ in range(4)]
    p = plans[0]
    batch = lib.Batch(plans)
    call = {'jk': lambda: torch.stack(p.get_jk_device(d, hermi=1)), 'grad': lambda: torch.stack(p.grad_jk_device(d)),
            'fill': lambda: p.int2e_s8(),
            'batch': lambda: torch.stack(sum(batch.get_jk_device([d] * 4), []))}[op]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        want = call()
        side.synchronize()
        lib.load().b200jk_debug_fail_alloc(nth)
        try:
            with pytest.raises(lib.B200JKError, match='lane of a stream set') as e:
                call()
            idle = side.query()
        finally:
            lib.load().b200jk_debug_fail_alloc(0)
        assert e.value.code == lib.B200JK_ECUDA and idle
        got = call()
        side.synchronize()
        assert float((got - want).abs().max()) < 1e-10 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize('nth', [1, 2, 5, 8, 9, 10, 16, 17])
def test_async_batch_after_a_failed_set_up(nth):
    """The synchronous batch call's set-up fails at one of its nine buffers, its
    seven streams or the scan storage: the asynchronous entry is refused on
    the host until a synchronous call has succeeded."""
    import torch
    from conftest import load_fixture
    from pyscf_b200 import lib
    if lib.device_count() == 0:
        pytest.skip('no GPU')
    f = load_fixture('h2o_vdz')
    d = torch.from_numpy(f['dm_rand'] + f['dm_rand'].T).cuda()
    plans = [lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13) for _ in range(2)]
    want = [p.get_jk_device(d, hermi=1) for p in plans]      # (their workspaces exist)
    batch = lib.Batch(plans)
    vj, vk = [torch.empty_like(d) for _ in plans], [torch.empty_like(d) for _ in plans]
    lib.load().b200jk_debug_fail_alloc(nth)
    try:
        with pytest.raises(lib.B200JKError):
            batch.get_jk_device([d, d])
    finally:
        lib.load().b200jk_debug_fail_alloc(0)
    with pytest.raises(lib.B200JKError, match='one b200jk_batch_get_jk call first') as e:
        batch.get_jk_device_async([d, d], vj, vk)
    assert e.value.code == lib.B200JK_EINVAL
    batch.get_jk_device([d, d])
    batch.get_jk_device_async([d, d], vj, vk)
    torch.cuda.synchronize()
    for j, k, (rj, rk) in zip(vj, vk, want):
        assert float((j - rj).abs().max()) < 1e-10 and float((k - rk).abs().max()) < 1e-10


@pytest.mark.parametrize('nth', [1, 3, 6])
def test_async_batch_after_a_failed_larger_build(nth):
    """A build of two densities on a plan of the batch fails while its
    workspace grows: the asynchronous entry sees that the workspace moved."""
    import numpy
    import torch
    from conftest import load_fixture
    from pyscf_b200 import lib
    if lib.device_count() == 0:
        pytest.skip('no GPU')
    f = load_fixture('h2o_vdz')
    h = f['dm_rand'] + f['dm_rand'].T
    d = torch.from_numpy(h).cuda()
    plans = [lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13) for _ in range(2)]
    batch = lib.Batch(plans)
    rj, rk = batch.get_jk_device([d, d])
    vj, vk = [torch.empty_like(d) for _ in plans], [torch.empty_like(d) for _ in plans]
    lib.load().b200jk_debug_fail_alloc(nth)
    try:
        with pytest.raises(lib.B200JKError) as e:
            plans[1].get_jk(numpy.array([h, h]), hermi=1)
        assert e.value.code == lib.B200JK_ENOMEM
    finally:
        lib.load().b200jk_debug_fail_alloc(0)
    with pytest.raises(lib.B200JKError, match='workspace moved') as e:
        batch.get_jk_device_async([d, d], vj, vk)
    assert e.value.code == lib.B200JK_EINVAL
    batch.get_jk_device([d, d])
    batch.get_jk_device_async([d, d], vj, vk)
    torch.cuda.synchronize()
    for got, want in zip(vj + vk, rj + rk):
        assert float((got - want).abs().max()) < 1e-10
