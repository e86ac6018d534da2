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


# More query tiles than a round of the workers (592) holds, for each kernel and each form of the workers: launches of any length overlap.
@pytest.mark.parametrize("B,H,S,D,kernel", [(60, 16, 128, 64, "KERNEL_WORKERS"), (21, 16, 320, 64, "KERNEL_WORKERS"), (9, 16, 1024, 64, "KERNEL_WORKERS"),
                                            (40, 16, 128, 128, "KERNEL_GENERAL"), (14, 16, 384, 128, "KERNEL_GENERAL")])
def test_long_launches_see_each_others_output(pkg, wl, torch_cuda, B, H, S, D, kernel):
    """A chain of calls, each with the output of the one before as its queries and keys, gives what the same calls give with a
    synchronisation between them."""
    torch = torch_cuda
    q8, _, v8, mask, amax = _tensors(wl, B, H, S, S, D, seed=S, valid=np.random.default_rng(S).integers(1, S + 1, B))
    param, desc = pkg.FMHAParamI8(*amax[:3], amax[2] / 4, 1.0), pkg.AttnDataDescriptor(B, S, H, D)
    plan = pkg.debug_plan(pkg.AttnDataDescriptorX(B, S, S, H, D))
    assert plan[0] == getattr(pkg, kernel) and B * H * -(-S // 128) > 592
    q, v, m = (torch.from_numpy(x).cuda() for x in (q8, v8, mask))
    results = []
    for wait in (True, False):
        x, bufs = q, [torch.zeros_like(q) for _ in range(12)]
        torch.cuda.synchronize()
        for o in bufs:
            pkg.FMHAInferI8(None, param, desc, x, x, v, m, o)
            x = o
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        results.append(bufs)
    for i, (a, b) in enumerate(zip(*results)):
        assert a.any() and torch.equal(a, b), f"call {i} of the chain read its input too early"
    assert pkg.device_status()[0] == pkg.OK


@pytest.mark.parametrize("what", ["few_rows", "policy", "policy_many", "policy_rounds"])
def test_buffers_rewritten_between_overlapping_launches(pkg, wl, torch_cuda, what):
    """One set of buffers, filled anew by every step's launches while the launches of the step before may still drain: the quantised
    query of a decoding step, the row statistics of a policy.  The outputs are those of steps with a synchronisation between them."""
    torch = torch_cuda
    B, H, Sq, Sk, D = {"few_rows": (3, 5, 1, 704, 128), "policy": (1, 5, 100, 320, 64), "policy_many": (30, 13, 100, 192, 64), "policy_rounds": (70, 13, 100, 192, 64)}[what]
    _, k8, v8, mask, amax = _tensors(wl, B, H, Sq, Sk, D, seed=Sq, valid=np.random.default_rng(B).integers(1, Sk, B))
    k, v, m = (torch.from_numpy(x).cuda() for x in (k8, v8, mask))
    desc, param = pkg.AttnDataDescriptorX(B, Sq, Sk, H, D), pkg.FMHAParamI8(*amax, 1.0)
    xs = [torch.randn((B, H, Sq, D), device="cuda") for _ in range(40)]
    q, scratch = torch.zeros((B, H, Sq, D), dtype=torch.int8, device="cuda"), torch.zeros(2 * B * H * Sq, device="cuda")
    results = []
    for wait in (True, False):
        outs = [torch.zeros_like(q) for _ in xs]
        torch.cuda.synchronize()
        for x, o in zip(xs, outs):
            pkg.quantize_f32(None, x, q)
            if what == "few_rows":
                pkg.FMHAInferI8Cross(None, param, desc, q, k, v, m, o)
            else:
                pkg.FMHAInferI8Policy(None, param, desc, q, k, v, m, o, pkg.POLICY_ROW, scratch)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        results.append([o.cpu().numpy() for o in outs])
    for i, (a, b) in enumerate(zip(*results)):
        assert np.array_equal(a, b), f"step {i} read what another step had left"
    assert pkg.device_status()[0] == pkg.OK


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    torch.cuda.set_device(0)
    return torch


# One cluster of 1, 2, 4, 8 and 16 CTAs; then the whole chip, where a warp has 0, 1, 4 (all kept in registers), 7 and 8 (one
# ring), 12 tiles of 1024 elements, with and without a remainder.  Up to 12 tiles a warp holds in registers and its ring; with 13 to 20
# tensor memory holds eight as well, with 21 and 33 the rest is read again, from the L2 and, beyond what that is asked to hold, from DRAM.
SWEEP = 148 * 8 * 1024
@pytest.mark.parametrize("n", [1, 3, 8192, 8193, 32771, 65536, 65537, 262144, 262147, 524288, 524289, SWEEP - 1, SWEEP, 4 * SWEEP + 1,
                               5 * SWEEP, 7 * SWEEP + 1023, 8 * SWEEP, 12 * SWEEP + 1025, 11 * SWEEP, 11 * SWEEP + 1024, 19 * SWEEP - 1, 20 * SWEEP + 2047,
                               33 * SWEEP + 5])
def test_quantize_sizes(pkg, oracle, torch_cuda, n):
    torch = torch_cuda
    x = np.random.default_rng(n).standard_normal(n, dtype=np.float32)
    for at in sorted({0, n // 2, n - 1}):                   # wherever the largest magnitude sits, it is found
        y = x.copy()
        y[at] = -7.5 - np.abs(x).max()
        out = torch.full((n + 64,), 0x5A, dtype=torch.int8, device="cuda")
        amax = torch.zeros(1, device="cuda")
        pkg.quantize_f32(None, torch.from_numpy(y).cuda(), out, amax, n=n)
        host = out.cpu().numpy()
        assert np.float32(amax.item()) == np.abs(y).max()
        assert np.array_equal(host[:n], oracle.quantize(y, np.abs(y).max())), (n, at)
        assert np.all(host[n:] == 0x5A)
    assert pkg.device_status()[0] == pkg.OK


@pytest.mark.parametrize("n", [5 * SWEEP + 1024, 6 * SWEEP + 3, 12 * SWEEP, 12 * SWEEP + 1024, 20 * SWEEP, 20 * SWEEP + 1024, 21 * SWEEP + 1, 27 * SWEEP + 7])
def test_quantize_sizes_around_what_a_warp_holds(pkg, oracle, torch_cuda, n):
    """Five tiles of a warp in registers, seven in its ring, eight in tensor memory: on and beyond each sum of them."""
    test_quantize_sizes(pkg, oracle, torch_cuda, n)


@pytest.mark.parametrize("n", [4099, 524289, 20 * SWEEP + 3])
@pytest.mark.parametrize("what", ["nan", "one_lane", "inf", "tiny", "huge", "zero"])
def test_quantize_values_that_are_no_ordinary_numbers(pkg, torch_cuda, n, what):
    """Elements that are no numbers, scales that are not finite or the largest there are: floor(x * scale + 0.5) limited to +-127 step by
    step in fp32, a NaN giving -127 (as the minimum and maximum of a number and a NaN are the number)."""
    torch = torch_cuda
    x = torch.randn(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    x[n // 3] = -6.5
    if what == "nan":
        x[::1237] = float("nan")
    elif what == "one_lane":         # one of the 32 lanes that share a tile of 1024 elements, another one in every tile
        tiles = torch.arange(n // 1024, device="cuda")
        x[1024 * tiles + 128 * (tiles % 8) + 4 * (tiles % 31)] = float("nan")
    elif what == "inf":
        x[n // 2], x[n - 1] = float("inf"), float("-inf")
    elif what == "tiny":
        x *= 1e-38                   # the scale is infinite
        x[::3] = 0.0
    elif what == "huge":
        x *= 5e37
    else:
        x.zero_()
    out, amax = torch.zeros(n, dtype=torch.int8, device="cuda"), torch.zeros(1, device="cuda")
    pkg.quantize_f32(None, x, out, amax)
    most = torch.nan_to_num(x, nan=0.0, posinf=float("inf"), neginf=float("-inf")).abs().max()
    scale = torch.tensor(127.0, device="cuda") / most if most > 0 else torch.zeros((), device="cuda")
    want = torch.nan_to_num(torch.floor(x * scale + 0.5), nan=-127.0, posinf=127.0, neginf=-127.0).clamp(-127, 127).to(torch.int8)
    assert amax.item() == most.item()
    assert torch.equal(out, want)
    assert pkg.device_status()[0] == pkg.OK


# The sizes that one cluster of 16 CTAs holds, on a device that has no room for one: from 256 tiles for 32 CTAs to 512 for 64.
@pytest.mark.parametrize("n", [262145, 262144 + 1023, 300007, 524288])
def test_quantize_without_clusters_of_16(pkg, oracle, torch_cuda, n):
    torch = torch_cuda
    x = np.random.default_rng(n).standard_normal(n, dtype=np.float32)
    x[n - 1] = 9.25
    out, amax = torch.full((n + 64,), 0x5A, dtype=torch.int8, device="cuda"), torch.zeros(1, device="cuda")
    on_gpu = torch.from_numpy(x).cuda()
    pkg.debug_quantize_whole_chip(None, on_gpu, out, amax, n=n)
    host = out.cpu().numpy()
    assert np.float32(amax.item()) == np.abs(x).max()
    assert np.array_equal(host[:n], oracle.quantize(x, np.abs(x).max())) and np.all(host[n:] == 0x5A)
    with pytest.raises(pkg.FmhaError):
        pkg.debug_quantize_whole_chip(None, on_gpu, out, amax, n=262144)
    assert pkg.device_status()[0] == pkg.OK


def test_quantize_calls_overlap_on_two_streams(pkg, oracle, torch_cuda):
    torch = torch_cuda
    n = 3 * SWEEP + 5
    xs = [torch.randn(n, device="cuda") * s for s in (1.0, 30.0)]
    want = [oracle.quantize(x.cpu().numpy(), float(x.abs().max())) for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    outs = [torch.empty(n, dtype=torch.int8, device="cuda") for _ in range(24)]
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        pkg.quantize_f32(streams[i % 2], xs[i % 2], o)
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        assert np.array_equal(o.cpu().numpy(), want[i % 2]), i
    assert pkg.device_status()[0] == pkg.OK


# Just beyond what one cluster holds: 65 and 74 CTAs, so that two calls fit on the chip side by side.
@pytest.mark.parametrize("apart", [1, 63, 64, 128])
def test_quantize_calls_in_flight_share_nothing(pkg, oracle, torch_cuda, apart):
    """Two captured calls, `apart` calls after one another, replayed on two streams at once, and eager calls on a third: however their
    kernels meet, each finds its own largest magnitude."""
    torch = torch_cuda
    sizes, scales = (524288 + 37, 74 * 8192 - 5, 600001), (1.0, 30.0, 0.05)
    xs = [torch.randn(n, device="cuda") * s for n, s in zip(sizes, scales)]
    outs = [torch.zeros(n, dtype=torch.int8, device="cuda") for n in sizes]
    amaxs = [torch.zeros(1, device="cuda") for _ in sizes]
    want = [torch.from_numpy(oracle.quantize(x.cpu().numpy(), float(x.abs().max()))).cuda() for x in xs]
    pkg.quantize_f32(None, xs[2], outs[2], amaxs[2])
    graphs = []
    for i in range(2):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[i]):
            pkg.quantize_f32(None, xs[i], outs[i], amaxs[i])
        for _ in range(apart - 1):
            pkg.quantize_f32(None, xs[2], outs[2], amaxs[2])
    streams = [torch.cuda.Stream() for _ in sizes]
    torch.cuda.synchronize()
    for _ in range(8):
        for o, a in zip(outs, amaxs):
            o.zero_()
            a.zero_()
        torch.cuda.synchronize()
        for _ in range(10):
            for i in range(2):
                with torch.cuda.stream(streams[i]):
                    graphs[i].replay()
            pkg.quantize_f32(streams[2], xs[2], outs[2], amaxs[2])
        torch.cuda.synchronize()
        for i in range(3):
            assert float(amaxs[i]) == float(xs[i].abs().max()) and torch.equal(outs[i], want[i]), i
    assert pkg.device_status()[0] == pkg.OK


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,B,H,Sk,valid", [
    (1, 1, 1, 64, None),                     # half a key tile, most warps and CTAs idle
    (1, 2, 3, 192, (1, 192)),                # one key only; half a tile behind a whole one
    (1, 3, 2, 1088, (1088, 0, 129)),         # a batch without any key: zeros
    (1, 1, 2, 8192, (8000,)),                # eight CTAs per head, several tiles per warp
    (1, 40, 16, 320, None),                  # many heads
    (2, 2, 2, 704, (640, 513)), (3, 2, 2, 1024, (900, 1024)), (4, 1, 3, 2048, None), (5, 2, 2, 448, (448, 77)),
    (7, 1, 2, 4096, (3001,)), (8, 3, 3, 640, (640, 64, 500)), (9, 1, 2, 512, None)])
@pytest.mark.parametrize("uint8_p", [False, True])
def test_few_query_rows(pkg, wl, oracle, torch_cuda, D, Sq, B, H, Sk, valid, uint8_p):
    torch = torch_cuda
    q8, k8, v8, mask, amax = _tensors(wl, B, H, Sq, Sk, D, seed=Sq * Sk + D, mask_p=0.1 if Sk > 192 else 0.0, valid=valid)
    want = oracle.q128(q8, k8, v8, mask, amax, p_levels=255 if uint8_p else 128)
    q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
    buf = torch.full((q8.size + 256,), 0x5A, dtype=torch.int8, device="cuda")
    desc, param = pkg.AttnDataDescriptorX(B, Sq, Sk, H, D), pkg.FMHAParamI8(*amax, 1.0)
    pkg.FMHAInferI8Cross(None, param, desc, q, k, v, m, buf[128:-128], uint8_p=uint8_p)
    st, words = pkg.device_status()
    assert st == pkg.OK, words
    host = buf.cpu().numpy()
    assert np.all(host[:128] == 0x5A) and np.all(host[-128:] == 0x5A)
    assert_parity(host[128:-128].reshape(q8.shape), want, f"Sq{Sq} B{B}H{H}Sk{Sk}D{D}")
    if B * H > 3:                            # a slice that begins inside a batch
        begin, count = 1, B * H - 2
        part = torch.zeros(count * Sq * D, dtype=torch.int8, device="cuda")
        view = [x.reshape(B * H, -1, D)[begin:begin + count].contiguous() for x in (q, k, v)]
        pkg.FMHAInferI8Cross(None, param, desc, *view, m, part, bh_begin=begin, bh_count=count, uint8_p=uint8_p)
        assert np.array_equal(part.cpu().numpy(), host[128:-128].reshape(B * H, -1)[begin:begin + count].ravel())


def test_the_line_of_the_few_rows_kernel(pkg, torch_cuda):
    """Five to eight rows: the forward kernels took 0.54 to 0.87 of its time at head_dim 128 and for a single key tile."""
    for D, Sq, Sk, few in [(64, 1, 64, True), (64, 4, 128, True), (64, 5, 128, False), (64, 8, 64, False), (64, 5, 192, True), (64, 8, 4096, True),
                           (64, 9, 4096, False), (128, 1, 64, True), (128, 4, 16384, True), (128, 5, 64, False), (128, 8, 4096, False)]:
        for B, H in ((1, 1), (16, 32)):
            desc = pkg.AttnDataDescriptorX(B, Sq, Sk, H, D)
            assert (pkg.debug_plan(desc)[0] == pkg.KERNEL_FEW_ROWS) == few, (D, Sq, Sk)
            assert pkg.debug_plan(desc, pkg.PLAN_CALIBRATION)[0] in (pkg.KERNEL_GENERAL, pkg.KERNEL_WORKERS)
            assert all(pkg.debug_plan(desc, policy) == (pkg.KERNEL_POLICY, 1, 0) for policy in (pkg.POLICY_ROW, pkg.POLICY_STATIC))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,B,H,Sk,valid", [(8, 70, 3, 128, None), (5, 300, 2, 64, None), (6, 3, 5, 192, (192, 1, 70))])
def test_five_to_eight_query_rows_on_either_side_of_the_line(pkg, wl, oracle, torch_cuda, D, Sq, B, H, Sk, valid):
    torch = torch_cuda
    q8, k8, v8, mask, amax = _tensors(wl, B, H, Sq, Sk, D, seed=Sq * Sk, mask_p=0.1, valid=valid)
    q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
    o = torch.full((q8.size + 256,), 0x5A, dtype=torch.int8, device="cuda")
    pkg.FMHAInferI8Cross(None, pkg.FMHAParamI8(*amax, 1.0), pkg.AttnDataDescriptorX(B, Sq, Sk, H, D), q, k, v, m, o[128:-128])
    assert pkg.device_status()[0] == pkg.OK
    host = o.cpu().numpy()
    assert np.all(host[:128] == 0x5A) and np.all(host[-128:] == 0x5A)
    assert_parity(host[128:-128].reshape(q8.shape), oracle.q128(q8, k8, v8, mask, amax))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("amax_scale", [1e-6, 1.0, 1e4])
def test_masked_keys_vanish_at_every_scale(pkg, wl, oracle, torch_cuda, D, amax_scale):
    """Masked keys are pushed out of the scores by the preset of the accumulator: whatever the scale of the scores, and
    where the masked keys hold the largest scores of all, they count for nothing.  Every pattern of the mask inside a tile."""
    torch = torch_cuda
    B, H, S = 6, 2, 448
    q8, k8, v8, mask, amax = _tensors(wl, B, H, S, S, D, seed=D)
    mask[0, 1:] = 1                                   # one key
    mask[1, :-1] = 1                                  # the last key
    mask[2, ::2] = 1
    mask[3, 100:300] = 1                              # a whole tile and the ends of two
    mask[4] = np.random.default_rng(0).random(S) < 0.97
    k8 = np.where(mask[:, None, :, None] != 0, np.sign(q8.mean(2, keepdims=True)).astype(np.int8) * 127, k8)
    v8 = np.where(mask[:, None, :, None] != 0, np.int8(127), v8)
    amax = (amax[0] * amax_scale, amax[1], amax[2], amax[2])
    q, k, v, m = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (q8, k8, v8, mask))
    o = torch.zeros_like(q)
    pkg.FMHAInferI8(None, pkg.FMHAParamI8(*amax, 1.0), pkg.AttnDataDescriptor(B, S, H, D), q, k, v, m, o)
    assert pkg.device_status()[0] == pkg.OK
    assert_parity(o.cpu().numpy(), oracle.q128(q8, np.ascontiguousarray(k8), np.ascontiguousarray(v8), mask, amax))


# Scores so small that all probabilities of a row are equal: masked keys still count for nothing.  Scales on both sides of the
# smallest factor from scores to exponents that the kernels work with (2^-100), where a masked key's preset alone would no longer
# vanish, and close to the smallest that a call accepts; on every kernel that presets masked keys, and on the one that does not.
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("c2", [2.0 ** -99.9, 2.0 ** -100.1, 2.0 ** -126, 2.0 ** -145])
@pytest.mark.parametrize("what,B,H,Sq,Sk", [("plain", 2, 3, 320, 320), ("many", 30, 13, 100, 192), ("few_rows", 2, 2, 4, 704), ("shared", 2, 16, 200, 1984),
                                            ("row", 2, 3, 320, 320), ("row", 30, 13, 100, 192), ("host", 6, 11, 640, 640)])
def test_masked_keys_vanish_at_the_smallest_scales(pkg, wl, oracle, torch_cuda, D, c2, what, B, H, Sq, Sk):
    torch = torch_cuda
    valid = np.random.default_rng(B).integers(1, Sk, B)
    q8, k8, v8, mask, amax = _tensors(wl, B, H, Sq, Sk, D, seed=D + Sk, mask_p=0.1, valid=valid)
    v8 = np.where(mask[:, None, :, None] != 0, np.int8(127), v8)                 # what masked keys would add shows
    each = float(np.sqrt(c2 * np.sqrt(D) * 127.0 ** 2 / np.log2(np.e)))          # q_amax and k_amax for that factor
    amax = (each, each, amax[2], amax[3])
    param = pkg.FMHAParamI8(*amax, 1.0)
    desc, desc_x = pkg.AttnDataDescriptor(B, Sk, H, D), pkg.AttnDataDescriptorX(B, Sq, Sk, H, D)
    want = (oracle.policy(q8, k8, v8, mask, (*amax, 1.0), oracle.POLICY_ROW) if what == "row" else oracle.q128(q8, k8, v8, mask, amax))
    if what == "host":
        host = [torch.from_numpy(x).pin_memory() for x in (q8, k8, v8, mask)]
        o = torch.zeros_like(host[0]).pin_memory()
        dirty = [torch.full_like(t, 111).pin_memory() for t in host[:3]]         # what the staging rows of keys that are not fetched hold
        pkg.FMHAInferI8Host(param, desc, *dirty, torch.zeros_like(host[3]), o)
        pkg.FMHAInferI8Host(param, desc, *host, o)
    else:
        q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
        o = torch.zeros_like(q)
        if what == "row":
            pkg.FMHAInferI8Policy(None, param, desc_x, q, k, v, m, o, pkg.POLICY_ROW, torch.zeros(2 * B * H * Sq, device="cuda"))
        else:
            pkg.FMHAInferI8Cross(None, param, desc_x, q, k, v, m, o)
    assert pkg.device_status()[0] == pkg.OK
    assert_parity(o.cpu().numpy(), want, f"{what} D{D} c2 {c2}")


# Calls at head_dim 64 with many query tiles run four workers to an SM: fewer units than workers, all workers busy, a last round with
# one worker, several rounds; key tiles half beyond the sequence, sequences without a key, a mask with holes in every tile.
@pytest.mark.parametrize("B,H,Sq,Sk,mask_p", [(50, 8, 64, 64, 0.0), (30, 13, 100, 192, 0.3), (37, 16, 128, 128, 0.0), (11, 9, 961, 448, 0.05)])
@pytest.mark.parametrize("what", ["plain", "uint8", "row", "static", "amax"])
def test_many_query_tiles_head_dim_64(pkg, wl, oracle, torch_cuda, B, H, Sq, Sk, mask_p, what):
    torch = torch_cuda
    valid = np.random.default_rng(B).integers(1, Sk + 1, B)
    valid[3] = 0
    valid[4] = Sk
    q8, k8, v8, mask, amax = _tensors(wl, B, H, Sq, Sk, 64, seed=B + Sk, mask_p=mask_p, valid=valid)
    q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
    desc, param = pkg.AttnDataDescriptorX(B, Sq, Sk, H, 64), pkg.FMHAParamI8(*amax, 0.25)
    assert pkg.debug_plan(desc)[0] == pkg.KERNEL_WORKERS and pkg.debug_plan(desc, pkg.PLAN_CALIBRATION)[0] == pkg.KERNEL_WORKERS
    o = torch.full((q8.size + 256,), 0x5A, dtype=torch.int8, device="cuda")
    scratch = torch.zeros(2 * B * H * Sq, device="cuda")
    if what == "amax":
        got = torch.zeros(1, device="cuda")
        pkg.calibrate_o_amax(None, param, desc, q, k, v, m, got)
        # the same arithmetic with a known scale: the largest output quantises to 127, and to no more with 1 % of head room
        tops = []
        for s in (1.0, 1.01):
            pkg.FMHAInferI8Cross(None, pkg.FMHAParamI8(*amax[:3], float(got) * s, 1.0), desc, q, k, v, m, o[128:-128])
            tops.append(int(o[128:-128].abs().max()))
        assert tops[0] == 127 and tops[1] in (125, 126), tops
        return
    if what in ("row", "static"):
        policy = pkg.POLICY_ROW if what == "row" else pkg.POLICY_STATIC
        pkg.FMHAInferI8Policy(None, param, desc, q, k, v, m, o[128:-128], policy, scratch)
        want = oracle.policy(q8, k8, v8, mask, (*amax, 0.25), oracle.POLICY_ROW if what == "row" else oracle.POLICY_STATIC)
    else:
        pkg.FMHAInferI8Cross(None, param, desc, q, k, v, m, o[128:-128], uint8_p=what == "uint8")
        want = oracle.q128(q8, k8, v8, mask, amax, p_levels=255 if what == "uint8" else 128)
    st, words = pkg.device_status()
    assert st == pkg.OK, words
    host = o.cpu().numpy()
    assert np.all(host[:128] == 0x5A) and np.all(host[-128:] == 0x5A)
    assert_parity(host[128:-128].reshape(q8.shape), want, what)


# Few query tiles and many keys: a query tile is shared by a cluster of 2, 4 or 8 CTAs.  Parts without a key, one live tile in all,
# holes, a sequence without any key, fewer tiles than they divide into evenly.
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,Sq,Sk,valid,mask_p", [
    (1, 2, 128, 1024, None, 0.0), (2, 1, 100, 2048, (130, 2048), 0.0), (3, 2, 300, 1088, (1, 0, 1025), 0.2), (1, 3, 9, 4096, None, 0.5),
    (2, 16, 200, 1984, (1984, 1201), 0.0), (1, 1, 640, 8192, (8100,), 0.0)])
@pytest.mark.parametrize("uint8_p", [False, True])
def test_few_query_tiles_share_their_keys(pkg, wl, oracle, torch_cuda, D, B, H, Sq, Sk, valid, mask_p, uint8_p):
    torch = torch_cuda
    q8, k8, v8, mask, amax = _tensors(wl, B, H, Sq, Sk, D, seed=Sq + Sk + D, mask_p=mask_p, valid=valid)
    want = oracle.q128(q8, k8, v8, mask, amax, p_levels=255 if uint8_p else 128)
    q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
    o = torch.full((q8.size + 256,), 0x5A, dtype=torch.int8, device="cuda")
    desc = pkg.AttnDataDescriptorX(B, Sq, Sk, H, D)
    assert pkg.debug_plan(desc)[0] == pkg.KERNEL_GENERAL and pkg.debug_plan(desc)[1] in (2, 4, 8) and pkg.debug_plan(desc)[2] == 0
    for _ in range(3):
        pkg.FMHAInferI8Cross(None, pkg.FMHAParamI8(*amax, 1.0), desc, q, k, v, m, o[128:-128], uint8_p=uint8_p)
    st, words = pkg.device_status()
    assert st == pkg.OK, words
    host = o.cpu().numpy()
    assert np.all(host[:128] == 0x5A) and np.all(host[-128:] == 0x5A)
    assert_parity(host[128:-128].reshape(q8.shape), want, f"B{B}H{H}Sq{Sq}Sk{Sk}D{D}")


# Host buffers: one, two and four chunks, fewer heads than chunks, copies (no padding, or pageable memory) and the fetching kernel (padding),
# a slice that begins and ends inside a batch.  Staging memory starts out dirty: the rows that are not fetched must not matter.
@pytest.mark.parametrize("B,H,S,D,valid,pinned", [
    (1, 1, 64, 64, None, True), (2, 2, 192, 128, (33, 192), True), (1, 3, 4096, 128, (1000,), True), (6, 11, 640, 64, (1, 0, 640, 320, 97, 96), True),
    (6, 11, 640, 64, (1, 0, 640, 320, 97, 96), False), (3, 7, 1024, 128, None, True)])
def test_host_buffers(pkg, wl, oracle, torch_cuda, B, H, S, D, valid, pinned):
    torch = torch_cuda
    q8, k8, v8, mask, amax = _tensors(wl, B, H, S, S, D, seed=S + D, valid=valid)
    param, desc = pkg.FMHAParamI8(*amax, 1.0), pkg.AttnDataDescriptor(B, S, H, D)
    host = [torch.from_numpy(x).pin_memory() if pinned else torch.from_numpy(x) for x in (q8, k8, v8, mask)]
    dirty = [torch.full_like(t, -127).pin_memory() for t in host[:3]]
    o = torch.zeros_like(host[0]).pin_memory() if pinned else torch.zeros_like(host[0])
    pkg.FMHAInferI8Host(param, desc, *dirty, torch.zeros_like(host[3]), o)
    pkg.FMHAInferI8Host(param, desc, *host, o)
    dev = [t.cuda() for t in host]
    want = torch.zeros_like(dev[0])
    pkg.FMHAInferI8(None, param, desc, *dev, want)
    want = want.cpu().numpy()
    # another division of the work than the whole call's may pick another kernel: equal up to ties
    assert_parity(o.numpy(), want, "host against device")
    assert_parity(o.numpy()[:, :, ::37], oracle.q128(q8, k8, v8, mask, amax)[:, :, ::37], "host against oracle")
    if B * H > 4:
        begin, count = 2, B * H - 3
        part = [t.reshape(B * H, S, D)[begin:begin + count].contiguous() for t in host[:3]]
        part = [t.pin_memory() for t in part] if pinned else part
        out = torch.zeros_like(part[0])
        pkg.FMHAInferI8HostSlice(param, desc, *part, host[3], out, begin, count)
        assert_parity(out.numpy(), want.reshape(B * H, S, D)[begin:begin + count], "slice")
    assert pkg.device_status()[0] == pkg.OK


def test_only_wholly_pinned_buffers_are_read_by_a_kernel(pkg, torch_cuda):
    """A kernel that reads host memory must find every byte of it pinned.  Only the decision is looked at; nothing is launched."""
    torch = torch_cuda
    B, H, S, D = 6, 11, 640, 64
    n, page = B * H * S * D, 4096
    desc, mask = pkg.AttnDataDescriptor(B, S, H, D), torch.ones((B, S), dtype=torch.int8)
    mask[:, :64] = 0                                     # so much padding that the kernel is worth it
    pinned = [torch.zeros(n + page, dtype=torch.int8).pin_memory() for _ in range(3)]
    q, k, v = (t[:n] for t in pinned)
    assert pkg.debug_host_fetch(desc, q, k, v, mask)
    assert pkg.debug_host_fetch(desc, pinned[0][page:], k, v, mask)                  # up to the end of its block
    assert not pkg.debug_host_fetch(desc, pinned[0][8:], k, v, mask)                 # not 16-byte aligned
    plain = np.zeros(n + 3 * page, np.int8)
    first = (plain.ctypes.data + page - 1) // page * page
    assert not pkg.debug_host_fetch(desc, q, first, v, mask)                         # pageable
    rt = torch.cuda.cudart()

    def with_registered(ranges):
        """The decision for q, k or v at `first`, with these byte ranges behind it registered."""
        try:
            done = []
            for begin, end in ranges:
                assert int(rt.cudaHostRegister(first + begin, end - begin, 0)) == 0
                done.append(begin)
            return [pkg.debug_host_fetch(desc, *(first if i == j else t for j, t in enumerate((q, k, v))), mask) for i in range(3)]
        finally:
            for begin in done:
                rt.cudaHostUnregister(first + begin)

    whole = (n + page - 1) // page * page
    assert with_registered([(0, whole)]) == [True] * 3
    assert with_registered([(0, whole - page)]) == [False] * 3                       # all but the end
    assert with_registered([(0, page), (whole - page, whole)]) == [False] * 3        # both ends, a hole between them


def test_a_mask_on_the_device_is_not_read_by_the_host(pkg, torch_cuda):
    """The choice between copies and the fetching kernel looks at the mask, unless the host cannot."""
    torch = torch_cuda
    desc, mask = pkg.AttnDataDescriptor(2, 256, 4, 64), torch.ones((2, 256), dtype=torch.int8)
    mask[:, :32] = 0
    q, k, v = (torch.zeros(2 * 4 * 256 * 64, dtype=torch.int8).pin_memory() for _ in range(3))
    assert pkg.debug_host_fetch(desc, q, k, v, mask) and pkg.debug_host_fetch(desc, q, k, v, mask.pin_memory())
    assert not pkg.debug_host_fetch(desc, q, k, v, mask.cuda())


def test_where_a_query_tile_is_shared(pkg, torch_cuda):
    """Either side of the lines: 12 query tiles of so many rows and key tiles, and 148 + 60."""
    for D, Sq, tiles, shared in [(64, 128, 5, False), (64, 128, 6, True), (128, 64, 5, False), (128, 64, 6, True), (128, 96, 6, False), (128, 96, 7, True), (128, 128, 7, False),
                                 (128, 128, 8, True), (64, 128, 64, True), (128, 128, 64, True)]:
        assert (pkg.debug_plan(pkg.AttnDataDescriptorX(1, Sq, 128 * tiles, 12, D))[1] > 1) == shared, (D, Sq, tiles)
    for D in (64, 128):
        for tiles, shared in [(5, False), (6, True)]:
            plan = pkg.debug_plan(pkg.AttnDataDescriptorX(1, 2048, 128 * tiles, 13, D))
            assert plan == ((pkg.KERNEL_GENERAL, 2, 1) if shared else (pkg.KERNEL_GENERAL, 1, 0)), (D, tiles)


# More query tiles than SMs: those of a last round of at most half the SMs are shared by pairs of CTAs.  148 + 2, 148 + 74 (the most) and
# 2 * 148 + 64 query tiles; the last of them beyond the sequence's end.  Where two whole rounds come first, the shared tiles belong to a
# sequence whose keys divide unevenly, leave one CTA of a pair without any, or leave none at all.
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,Sq,Sk,valid,mask_p,rounds", [
    (3, 10, 600, 1088, (1088, 650, 0), 0.0, 1), (2, 37, 300, 1024, (1000, 129), 0.0, 1),
    (2, 12, 1900, 1280, (1280, 700), 0.1, 2), (2, 12, 1900, 1280, (900, 100), 0.0, 2), (2, 12, 1900, 1280, (1280, 0), 0.0, 2)])
def test_pairs_share_the_last_round(pkg, wl, oracle, torch_cuda, D, B, H, Sq, Sk, valid, mask_p, rounds):
    torch = torch_cuda
    q8, k8, v8, mask, amax = _tensors(wl, B, H, Sq, Sk, D, seed=Sq + Sk + D, mask_p=mask_p, valid=valid)
    want = oracle.q128(q8, k8, v8, mask, amax)
    q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
    o = torch.full((q8.size + 256,), 0x5A, dtype=torch.int8, device="cuda")
    desc = pkg.AttnDataDescriptorX(B, Sq, Sk, H, D)
    assert pkg.debug_plan(desc) == (pkg.KERNEL_GENERAL, 2, rounds)
    for _ in range(3):
        pkg.FMHAInferI8Cross(None, pkg.FMHAParamI8(*amax, 1.0), desc, q, k, v, m, o[128:-128])
    st, words = pkg.device_status()
    assert st == pkg.OK, words
    host = o.cpu().numpy()
    assert np.all(host[:128] == 0x5A) and np.all(host[-128:] == 0x5A)
    assert_parity(host[128:-128].reshape(q8.shape), want, f"B{B}H{H}Sq{Sq}Sk{Sk}D{D}")


@pytest.mark.parametrize("o_scale", [4.0, 0.3, 0.1, 1e-4])
@pytest.mark.parametrize("D,Sk", [(128, 128), (128, 384), (64, 192)])
def test_outputs_on_both_sides_of_the_clamp(pkg, wl, oracle, torch_cuda, D, Sk, o_scale):
    """No output, a few rows', most of them and all of them beyond +-127.  (A row with one key repeats its V8 / o_scale: above
    127 for |v8| > 38 at o_scale 0.3, one standard deviation of it; and never above 127 / 4 + 1 at o_scale 4.)"""
    torch = torch_cuda
    q8, k8, v8, mask, amax = _tensors(wl, 3, 5, Sk, Sk, D, seed=Sk + D, valid=[Sk, 1, Sk - 3])
    amax = amax[:3] + (amax[2] * o_scale,)
    q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
    o = torch.full_like(q, 77)
    pkg.FMHAInferI8(None, pkg.FMHAParamI8(*amax, 1.0), pkg.AttnDataDescriptor(3, Sk, 5, D), q, k, v, m, o)
    torch.cuda.synchronize()
    got = o.cpu().numpy()
    assert_parity(got, oracle.q128(q8, k8, v8, mask, amax), f"o_scale {o_scale}")
    assert np.abs(got.astype(int)).max() <= 127
    assert (np.abs(got.astype(int)) == 127).any() == (o_scale < 0.5)
    assert pkg.device_status()[0] == pkg.OK


# Key tiles with unmasked keys in one half only, which the workers process as 64 keys.  Lengths on either side of half a tile, sequences
# that end in half a tile, an open lower or upper half with and without masked keys in it, alone and beside whole tiles; in the workers'
# two forms (up to three key tiles and more), the other kernels, and the launches of a whole-row policy.
HALVES = {
    "lengths": lambda Sk, b, rng: np.arange(Sk) >= [1, 63, 64, 65, 127, 128, 129, 192, 193, 255, Sk - 64, Sk - 1, Sk][b % 13],
    "upper": lambda Sk, b, rng: (np.arange(Sk) % 128 < 64) | (np.arange(Sk) % 5 == b % 7),
    "either": lambda Sk, b, rng: ((np.arange(Sk) // 64) % 4 != b % 4) & ((np.arange(Sk) // 64) % 3 != b % 3) | (rng.random(Sk) < 0.1 * (b % 2)),
}
@pytest.mark.parametrize("B,H,Sq,Sk,D", [(104, 16, 64, 64, 64), (104, 8, 256, 256, 64), (52, 16, 320, 320, 64), (52, 8, 130, 576, 64),
                                         (13, 2, 320, 320, 64), (13, 2, 320, 320, 128), (13, 1, 100, 576, 64), (13, 1, 257, 576, 128), (13, 4, 1, 576, 128)])
@pytest.mark.parametrize("how", sorted(HALVES))
def test_half_tiles(pkg, wl, oracle, torch_cuda, B, H, Sq, Sk, D, how):
    torch = torch_cuda
    q8, k8, v8, _, (qa, ka, va, _) = _tensors(wl, B, H, Sq, Sk, D, seed=Sk + D + B)
    # A probability at a rounding boundary moves an output by s_max * v_amax / o_amax (static), at most v_amax / o_amax (the others) of
    # its steps: with o_amax = v_amax by one, as assert_parity expects.  (With the o_amax of _tensors, v_amax / 8, by up to four.)
    amax = (qa, ka, va, va)
    rng = np.random.default_rng(Sk)
    mask = np.stack([HALVES[how](Sk, b, rng) for b in range(B)]).astype(np.int8)
    q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
    o = torch.full_like(q, 0x5A)
    param, desc = pkg.FMHAParamI8(*amax, 0.5), pkg.AttnDataDescriptorX(B, Sq, Sk, H, D)
    pkg.FMHAInferI8Cross(None, param, desc, q, k, v, m, o)
    got = o.cpu().numpy()
    # a few heads of every batch against the oracle, all of them against the CUDA-core kernel
    ref = torch.empty_like(o)
    pkg.debug_simt_x(None, param, desc, q, k, v, m, ref)
    assert_parity(got, ref.cpu().numpy(), "against the CUDA-core kernel")
    some = slice(0, 13)
    want = oracle.q128(q8[some, :1], k8[some, :1], v8[some, :1], mask[some], amax)
    assert_parity(got[some, :1], want, "against the oracle")
    if Sq > 8:
        scratch = torch.zeros(2 * B * H * Sq, device="cuda")
        for policy, which in ((pkg.POLICY_ROW, oracle.POLICY_ROW), (pkg.POLICY_STATIC, oracle.POLICY_STATIC)):
            pkg.FMHAInferI8Policy(None, param, desc, q, k, v, m, o, policy, scratch)
            want = oracle.policy(q8[some, :1], k8[some, :1], v8[some, :1], mask[some], (*amax, 0.5), which)
            assert_parity(o.cpu().numpy()[some, :1], want, f"policy {policy}")
    assert pkg.device_status()[0] == pkg.OK


# Many query tiles, most of whose sequences have no unmasked key at all: behind the last open one a worker meets five to seven empty
# ones in a row, more than it has room to announce.
@pytest.mark.parametrize("what", ["forward", "row", "static", "amax"])
@pytest.mark.parametrize("open_batches", [0, 1, 592, 600])
def test_rows_of_empty_units(pkg, wl, oracle, torch_cuda, open_batches, what):
    torch = torch_cuda
    B, H, Sq, Sk, D = 4200, 1, 70, 64, 64
    q8, k8, v8, _, (qa, ka, va, _) = _tensors(wl, B, H, Sq, Sk, D, seed=7)
    mask = np.ones((B, Sk), np.int8)
    mask[:open_batches, :50] = 0
    q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
    o = torch.full_like(q, 0x5A)
    param, desc = pkg.FMHAParamI8(qa, ka, va, va, 0.5), pkg.AttnDataDescriptorX(B, Sq, Sk, H, D)
    assert pkg.debug_plan(desc)[0] == pkg.KERNEL_WORKERS
    n = max(1, open_batches)
    if what == "amax":
        most = torch.zeros(1, device="cuda")
        pkg.calibrate_o_amax(None, param, desc, q, k, v, m, most)
        o32, _ = oracle.fp32_attention(*(x[:n].astype(np.float32) * np.float32(a / 127) for x, a in ((q8, qa), (k8, ka), (v8, va))), mask[:n])
        want = float(np.abs(o32).max()) if open_batches else 0.0
        assert abs(most.item() - want) <= 0.02 * want
    else:
        if what == "forward":
            pkg.FMHAInferI8Cross(None, param, desc, q, k, v, m, o)
            want = oracle.q128(q8[:n], k8[:n], v8[:n], mask[:n], (qa, ka, va, va))
        else:
            policy, which = (pkg.POLICY_ROW, oracle.POLICY_ROW) if what == "row" else (pkg.POLICY_STATIC, oracle.POLICY_STATIC)
            pkg.FMHAInferI8Policy(None, param, desc, q, k, v, m, o, policy, torch.zeros(2 * B * H * Sq, device="cuda"))
            want = oracle.policy(q8[:n], k8[:n], v8[:n], mask[:n], (qa, ka, va, va, 0.5), which)
        got = o.cpu().numpy()
        assert_parity(got[:n], want, what)
        assert not got[open_batches:].any()
    assert pkg.device_status()[0] == pkg.OK


# Factors from scores to exponents at which a difference of one in the scores is anything from a few per cent to everything: 2^(-c2) per
# unit.  (Not chosen at a boundary of the rounding of 128, 255 or 127 times 2^(-c2 * n): every key of a row has one of a few scores.)
LARGE_SCALES = [0.0031, 0.077, 0.317, 0.931, 2.37, 3.13, 10.7, 49.3, 71.9, 1.3e4, 1.1e15, 1.7e31]
LARGE_SCALE_CALLS = {  # B, H, Sq, Sk, D -> the kernel that runs it
    (2, 3, 1, 704, 128): "KERNEL_FEW_ROWS", (2, 3, 3, 704, 64): "KERNEL_FEW_ROWS", (1, 3, 200, 1024, 128): "KERNEL_GENERAL",
    (8, 20, 256, 512, 128): "KERNEL_GENERAL", (2, 3, 70, 448, 64): "KERNEL_GENERAL", (40, 12, 256, 320, 64): "KERNEL_WORKERS",
    (18, 16, 256, 640, 64): "KERNEL_WORKERS", (2, 3, 70, 128, 64): "KERNEL_GENERAL", (2, 3, 70, 128, 128): "KERNEL_GENERAL"}


@pytest.mark.parametrize("c2", LARGE_SCALES)
@pytest.mark.parametrize("B,H,Sq,Sk,D", sorted(LARGE_SCALE_CALLS))
def test_large_score_scales(pkg, wl, oracle, torch_cuda, B, H, Sq, Sk, D, c2):
    """Scores that are small whole numbers, so that a row's keys share their maximum with others of the same tile and of other tiles at
    every scale, up to the largest that a call takes."""
    torch = torch_cuda
    rng = np.random.default_rng(Sk + D)
    q8 = np.zeros((B, H, Sq, D), np.int8)
    at = rng.integers(0, D, (B, H, Sq, 4))
    np.put_along_axis(q8, at, rng.choice(np.array([-1, 1], np.int8), at.shape), -1)
    k8 = rng.choice(np.array([-1, 0, 0, 0, 1], np.int8), (B, H, Sk, D))
    v8 = np.clip(np.rint(rng.standard_normal((B, H, Sk, D)) * 40), -127, 127).astype(np.int8)
    mask = (np.arange(Sk)[None, :] >= rng.integers(Sk // 2, Sk + 1, B)[:, None]).astype(np.int8)
    each = float(np.sqrt(c2 * np.sqrt(D) * 127.0 ** 2 / np.log2(np.e)))          # q_amax and k_amax for that factor
    # o_amax: where a level lies at a rounding boundary, all of a row's equal keys, 20 at the most here, move by one.  With the static
    # scale that is v_amax / o_amax * s_max / 127 times the sum of their values (standard deviation 40 sqrt(20) = 180): 1.3 v_amax / o_amax for the
    # largest s_max, three times that in the worst of some thousand rows; 2 with this o_amax.
    amax = (each, each, 3.0, 6.0)
    # s_max: nine tenths of the largest probability.  (With all of it, rows of two equal keys would have 127 / 2 to round.)
    score = np.einsum("bid,bjd->bij", q8[:, 0].astype(np.float32), k8[:, 0].astype(np.float32)).astype(np.float64)
    score[np.broadcast_to(mask[:, None, :] != 0, score.shape)] = -np.inf
    s_max = 0.9 / float(np.exp2(c2 * (score - score.max(-1, keepdims=True))).sum(-1).min())
    q, k, v, m = (torch.from_numpy(x).cuda() for x in (q8, k8, v8, mask))
    o, ref = torch.full_like(q, 0x5A), torch.empty_like(q)
    param, desc = pkg.FMHAParamI8(*amax, s_max), pkg.AttnDataDescriptorX(B, Sq, Sk, H, D)
    assert pkg.debug_plan(desc)[0] == getattr(pkg, LARGE_SCALE_CALLS[(B, H, Sq, Sk, D)])
    pkg.FMHAInferI8Cross(None, param, desc, q, k, v, m, o)
    got = o.cpu().numpy()
    assert_parity(got[:, :1], oracle.q128(q8[:, :1], k8[:, :1], v8[:, :1], mask, amax), "against the oracle")
    pkg.debug_simt_x(None, param, desc, q, k, v, m, ref)
    assert_parity(got, ref.cpu().numpy(), "against the CUDA-core kernel")
    pkg.FMHAInferI8Cross(None, param, desc, q, k, v, m, o, uint8_p=True)
    assert_parity(o.cpu().numpy()[:, :1], oracle.q128(q8[:, :1], k8[:, :1], v8[:, :1], mask, amax, p_levels=255), "255 levels")
    scratch = torch.zeros(2 * B * H * Sq, device="cuda")
    for policy, which in ((pkg.POLICY_ROW, oracle.POLICY_ROW), (pkg.POLICY_STATIC, oracle.POLICY_STATIC)):
        pkg.FMHAInferI8Policy(None, param, desc, q, k, v, m, o, policy, scratch)
        assert_parity(o.cpu().numpy()[:, :1], oracle.policy(q8[:, :1], k8[:, :1], v8[:, :1], mask, (*amax, s_max), which), f"policy {policy}")
    assert pkg.device_status()[0] == pkg.OK


# Query tiles of S keys on either side of the line between the two head_dim-64 kernels (on 148 SMs), and calibration's own line.
@pytest.mark.parametrize("units,S,forward,calibration", [
    (100, 64, "GENERAL", "GENERAL"), (296, 128, "WORKERS", "WORKERS"), (296, 256, "GENERAL", "WORKERS"), (520, 256, "WORKERS", "WORKERS"),
    (740, 256, "GENERAL", "WORKERS"), (1184, 256, "WORKERS", "WORKERS"), (444, 512, "GENERAL", "WORKERS"), (592, 1024, "WORKERS", "WORKERS"),
    (288, 1024, "GENERAL", "GENERAL"), (1184, 2048, "WORKERS", "WORKERS")])
def test_line_between_the_kernels_of_head_dim_64(pkg, torch_cuda, units, S, forward, calibration):
    if torch_cuda.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the line lies elsewhere on another number of SMs")
    desc = pkg.AttnDataDescriptorX(units * 128 // max(S, 128), S, S, 1, 64)
    assert pkg.debug_plan(desc)[0] == getattr(pkg, "KERNEL_" + forward)
    assert pkg.debug_plan(desc, pkg.PLAN_CALIBRATION)[0] == getattr(pkg, "KERNEL_" + calibration)


# Single key tiles in less than two rounds of SMs, and query tiles too many for clusters of four: either side of the lines (on 148 SMs).
@pytest.mark.parametrize("H,Sq,Sk,D,kernel,parts", [
    (160, 128, 128, 64, "GENERAL", 1), (295, 128, 128, 64, "GENERAL", 1), (160, 128, 64, 64, "WORKERS", 1), (32, 128, 768, 64, "GENERAL", 4), (37, 128, 896, 64, "GENERAL", 1),
    (37, 128, 1024, 64, "GENERAL", 2), (72, 128, 896, 64, "GENERAL", 1), (60, 128, 1152, 128, "GENERAL", 1), (60, 128, 1280, 128, "GENERAL", 2)])
def test_lines_of_single_tiles_and_of_pairs(pkg, torch_cuda, H, Sq, Sk, D, kernel, parts):
    if torch_cuda.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines lie elsewhere on another number of SMs")
    assert pkg.debug_plan(pkg.AttnDataDescriptorX(1, Sq, Sk, H, D))[:2] == (getattr(pkg, "KERNEL_" + kernel), parts)
