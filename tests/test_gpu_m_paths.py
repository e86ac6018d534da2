"""GPU tests of the choices that depend on a call's size: each at the sizes where it can go wrong, against the CPU oracle."""
import numpy as np
import pytest

from _util import assert_parity

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]


def _tensors(wl, B, H, Sq, Sk, D, seed, mask_p=0.0, valid=None):
    rng = np.random.Generator(np.random.Philox(key=seed))
    q8, qa = wl.quantize_np(rng.standard_normal((B, H, Sq, D), dtype=np.float32))
    k8, ka = wl.quantize_np(rng.standard_normal((B, H, Sk, D), dtype=np.float32))
    v8, va = wl.quantize_np(rng.standard_normal((B, H, Sk, D), dtype=np.float32))
    mask = (rng.random((B, Sk)) < mask_p).astype(np.int8)
    if valid is not None:
        mask |= (np.arange(Sk)[None, :] >= np.asarray(valid)[:, None]).astype(np.int8)
    keys = max(1, int((mask == 0).sum(1).min()))
    return q8, k8, v8, mask, (qa, ka, va, min(va, 6.0 * float(np.sqrt(np.e / keys))))


@pytest.mark.parametrize("S,D", [(64, 64), (320, 128)])
def test_back_to_back_calls_see_each_others_output(pkg, wl, torch_cuda, S, D):
    """Short launches start while the launch before them drains: a chain of dependent calls gives what the same calls
    give with a synchronisation between them."""
    torch = torch_cuda
    q8, k8, v8, mask, amax = _tensors(wl, 1, 3, S, S, D, seed=S)
    param, desc = pkg.FMHAParamI8(*amax, 1.0), pkg.AttnDataDescriptor(1, S, 3, D)
    q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
    results = []
    for wait in (True, False):
        x, bufs = q, [torch.zeros_like(q) for _ in range(40)]
        torch.cuda.synchronize()
        for o in bufs:
            pkg.FMHAInferI8(None, param, desc, x, k, v, m, o)
            x = o
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        results.append([b.cpu().numpy() for b in bufs])
    for i, (a, b) in enumerate(zip(*results)):
        assert np.array_equal(a, b), f"call {i} of the chain read its input too early"
    assert pkg.device_status()[0] == pkg.OK


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    torch.cuda.set_device(0)
    return torch
