"""Device calls on PyTorch's default stream: the engine reads tensors that work
queued on that stream has yet to write."""
import pytest

from conftest import load_fixture

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.fixture(scope='module')
def setup():
    import torch
    from pyscf_b200 import lib
    if lib.device_count() == 0:
        pytest.skip('no GPU')
    f = load_fixture('h2o_vdz')
    d = torch.from_numpy(f['dm_rand'] + f['dm_rand'].T).cuda()
    plan = lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13)
    batch = lib.Batch([lib.Plan(f['atm'], f['bas'], f['env'], direct_scf_tol=1e-13) for _ in range(2)])
    return d, plan, batch


def _late(d):
    """A copy of d that the default stream writes after 20 ms of other work."""
    import torch
    out = torch.zeros_like(d)
    torch.cuda.synchronize()
    torch.cuda._sleep(int(20e-3 * 1.9e9))
    out.copy_(d)
    return out


@pytest.mark.parametrize('op', ['jk', 'gradjk', 'force', 'batch', 'batch_async'])
def test_default_stream_order(setup, op):
    import torch
    d, plan, batch = setup
    assert torch.cuda.current_stream() == torch.cuda.default_stream()
    out = [torch.empty_like(d) for _ in range(4)]

    def batch_async(x):
        batch.get_jk_device_async([x, x], out[:2], out[2:])
        return torch.stack(out)     # queued on the default stream behind the build
    call = {'jk': lambda x: torch.stack(plan.get_jk_device(x, hermi=1)),
            'gradjk': lambda x: torch.stack(plan.grad_jk_device(x)),
            'force': lambda x: plan.grad_contract(x),
            'batch': lambda x: torch.stack(sum(batch.get_jk_device([x, x]), [])),
            'batch_async': batch_async}[op]
    batch.get_jk_device([d, d])
    torch.cuda.synchronize()
    want = call(d).clone()
    torch.cuda.synchronize()
    if op == 'batch_async':
        for o in out:
            o.zero_()
    got = call(_late(d))
    torch.cuda.synchronize()
    assert float((got - want).abs().max()) < TOL * max(1.0, float(want.abs().max()))
