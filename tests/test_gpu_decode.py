"""Decode attention on the GPU through the C ABI against the CPU oracle."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from helpers_gpu import dev, pos_tensor, poisoned_cache

pytestmark = pytest.mark.gpu
AD, GQA = 256, 6
SCALE = 1.0 / 16.0


@pytest.fixture(autouse=True, params=[1, 2, 3, 4], ids=["mma", "tc", "ws", "wt"])
def decode_kernel(request, q27):
    """Every test of this module runs on every split-K kernel (warp-MMA, tcgen05, warp-specialised, warp-specialised with P V on tcgen05)."""
    q27.set_decode_kernel(request.param)
    yield request.param
    q27.set_decode_kernel(0)


def run_decode(q27, orc, T, nkvh, n, n_ctx=None, seed_shift=0, check=True, q8_1=False):
    from qwen27_engine_b200 import synth
    nqh = nkvh * GQA
    n_ctx = n_ctx or n + 11
    qn, qg, kf, vf = synth.decode_inputs(T, nqh, nkvh, n, start_kv=seed_shift)
    kc_ref, vc_ref = orc.fill_cache(kf, vf, n_ctx)
    kc = poisoned_cache(q27, kc_ref, nkvh, n_ctx, n)
    vc = poisoned_cache(q27, vc_ref, nkvh, n_ctx, n)
    o = torch.full((T, nqh, AD), float("nan"), device="cuda")
    q27.attn_decode(dev(qn), dev(qg), kc, vc, o, None, None, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx)
    torch.cuda.synchronize()
    out = o.cpu().numpy()
    if check:
        ref = orc.attn_ref(qn, qg, kc_ref, vc_ref, n - T, SCALE, nkvh, n_ctx)
        assert_close(out, ref, "decode T=%d nkvh=%d n=%d" % (T, nkvh, n))
    return out, (qn, qg, kc, vc, kc_ref, vc_ref)


def test_config1_cpu_checkable(q27, orc):
    """1 query token, 24 Q / 4 KV heads, KV length 1024."""
    run_decode(q27, orc, 1, 4, 1024)
    assert q27.device_status() == 0


@pytest.mark.parametrize("T", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [4, 5, 7, 33, 63, 64, 65, 100, 127, 128, 129, 1000, 4096, 4100, 9472, 9473, 20011])
def test_decode_depths(q27, orc, T, n):
    if n < T:
        pytest.skip("fewer positions than query tokens")
    run_decode(q27, orc, T, 2, n)


@pytest.mark.parametrize("nkvh", [1, 2, 4])
def test_decode_head_counts(q27, orc, nkvh):
    run_decode(q27, orc, 4, nkvh, 3000)
    assert q27.device_status() == 0


def test_config2_spec_verify_32k(q27, orc):
    """4 query tokens (causal inside the block), 24 Q / 4 KV heads, q8_0 KV length 32,768."""
    run_decode(q27, orc, 4, 4, 32768)


def test_config3_long_context(q27, orc):
    for n in (30000, 100000, 150000):
        run_decode(q27, orc, 4, 4, n, n_ctx=n + 8)
    assert q27.device_status() == 0


def test_causal_inside_the_block(q27, orc):
    """Token t must not see the K/V of tokens t+1..: changing them leaves its output unchanged."""
    T, nkvh, n = 4, 1, 500
    out, (qn, qg, kc, vc, kc_ref, vc_ref) = run_decode(q27, orc, T, nkvh, n)
    kc2, vc2 = kc.clone(), vc.clone()
    n_ctx = n + 11
    # overwrite the last row (position n-1, visible to the last token only)
    kc2[: n_ctx * AD].view(n_ctx, AD)[n - 1] = 77
    vc2[: n_ctx * AD].view(n_ctx, AD)[n - 1] = 99
    o2 = torch.empty((T, nkvh * GQA, AD), device="cuda")
    q27.attn_decode(dev(qn), dev(qg), kc2, vc2, o2, None, None, pos_tensor(n - T), T, SCALE, nkvh * GQA, nkvh, n_ctx)
    torch.cuda.synchronize()
    o2 = o2.cpu().numpy()
    assert np.array_equal(o2[:3], out[:3]) and not np.array_equal(o2[3], out[3])


def test_run_twice_bitwise(q27, orc):
    a, _ = run_decode(q27, orc, 4, 4, 12345, check=False)
    b, _ = run_decode(q27, orc, 4, 4, 12345, check=False)
    assert np.array_equal(a, b)


def test_q8_1_epilogue(q27, orc):
    """With xq the result leaves as q8_1: exactly the oracle's q8_1 of the kernel's own f32 result."""
    T, nkvh, n = 4, 2, 2000
    nqh = nkvh * GQA
    out, (qn, qg, kc, vc, _, _) = run_decode(q27, orc, T, nkvh, n)
    xq = torch.zeros((T, nqh, AD), dtype=torch.int8, device="cuda")
    xd = torch.zeros((T * nqh * 8,), dtype=torch.float32, device="cuda")
    q27.attn_decode(dev(qn), dev(qg), kc, vc, None, xq, xd, pos_tensor(n - T), T, SCALE, nqh, nkvh, n + 11)
    torch.cuda.synchronize()
    rq, rd = orc.q8_1(out.reshape(-1))
    assert np.array_equal(xq.cpu().numpy().reshape(-1), rq) and np.array_equal(xd.cpu().numpy(), rd)


@pytest.mark.parametrize("n,cuts", [(1000, [0, 512, 1000]), (5000, [0, 1280, 2560, 3840, 5000]), (300, [0, 64, 300])])
def test_kv_length_partials_merge(q27, orc, n, cuts):
    """One sequence split by KV length (each slice a cache of its own, as on separate GPUs):
    per-slice partials + the log-sum-exp merge = the whole."""
    from qwen27_engine_b200 import synth
    T, nkvh = 4, 2
    nqh = nkvh * GQA
    qn, qg, kf, vf = synth.decode_inputs(T, nqh, nkvh, n)
    parts, refs = [], []
    full_k, full_v = orc.fill_cache(kf, vf, n)
    for lo, hi in zip(cuts, cuts[1:]):
        n_ctx = hi - lo + 3
        kc_ref, vc_ref = orc.fill_cache(kf[:, lo:hi], vf[:, lo:hi], n_ctx)
        kc = poisoned_cache(q27, kc_ref, nkvh, n_ctx, hi - lo)
        vc = poisoned_cache(q27, vc_ref, nkvh, n_ctx, hi - lo)
        part = torch.full((T, nqh, 258), float("nan"), device="cuda")
        q27.attn_decode_partial(dev(qn), kc, vc, part, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx, lo, hi - lo)
        parts.append(part)
        refs.append(orc.attn_partial(qn, full_k, full_v, n - T, SCALE, nkvh, n, lo, hi))
    allp = torch.stack(parts).contiguous()
    o = torch.empty((T, nqh, AD), device="cuda")
    q27.lse_merge(allp, len(parts), T * nqh * 258, T * nqh, dev(qg), o)
    torch.cuda.synchronize()
    whole = orc.attn_ref(qn, qg, full_k, full_v, n - T, SCALE, nkvh, n)
    assert_close(o.cpu().numpy(), whole, "merged slices")
    # each partial, normalised on its own, against the oracle's partial
    for part, ref in zip(parts, refs):
        a = part.cpu().numpy()
        live = ref[..., 1] > 0
        assert np.array_equal(a[..., 1] > 0, live)
        ya = a[..., 2:][live] / a[..., 1:2][live]
        yr = ref[..., 2:][live] / ref[..., 1:2][live]
        assert_close(ya, yr, "slice partial")
        lse_a = a[..., 0][live] + np.log(a[..., 1][live])
        lse_r = ref[..., 0][live] + np.log(ref[..., 1][live])
        assert np.abs(lse_a - lse_r).max() < 2e-3
    assert q27.device_status() == 0


def test_lse_merge_generic(q27, orc):
    rng = np.random.default_rng(5)
    nparts, rows = 7, 50
    parts = rng.standard_normal((nparts, rows, 258)).astype(np.float32)
    parts[..., 1] = np.abs(parts[..., 1]) + 0.1
    parts[3, :, 0] = -1e30   # an empty partial is neutral
    parts[3, :, 1:] = 0
    qg = rng.standard_normal((rows, 512)).astype(np.float32)
    ref = orc.lse_merge(parts, qg)
    o = torch.empty((rows, AD), device="cuda")
    q27.lse_merge(dev(parts), nparts, rows * 258, rows, dev(qg), o)
    torch.cuda.synchronize()
    assert np.abs(o.cpu().numpy() - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max())
    ref2 = orc.lse_merge(parts, None)
    q27.lse_merge(dev(parts), nparts, rows * 258, rows, None, o)
    torch.cuda.synchronize()
    assert np.abs(o.cpu().numpy() - ref2).max() <= 1e-5 * max(1.0, np.abs(ref2).max())


@pytest.mark.parametrize("T,nkvh,n", [(4, 2, 777), (1, 1, 5), (4, 4, 64), (3, 2, 129), (2, 1, 4100), (4, 4, 32768)])
def test_f16_kv_cache(q27, orc, T, nkvh, n):
    """The f16 KV cache variant of the decode kernel (config: the 32,768 spec-verify case also with f16 KV)."""
    from qwen27_engine_b200 import synth
    nqh = nkvh * GQA
    qn, qg, kf, vf = synth.decode_inputs(T, nqh, nkvh, n)
    kc_ref, vc_ref = orc.fill_cache(kf, vf, n + 5, q8=False)
    o = torch.empty((T, nqh, AD), device="cuda")
    try:
        q27.attn_decode(dev(qn), dev(qg), poisoned_cache(q27, kc_ref, nkvh, n + 5, n, False),
                        poisoned_cache(q27, vc_ref, nkvh, n + 5, n, False), o, None, None, pos_tensor(n - T), T, SCALE,
                        nqh, nkvh, n + 5, q8=False)
    except q27.Q27Error as e:
        assert e.code == q27.UNSUPPORTED
        pytest.skip("f16 KV decode not built: " + str(e))
    torch.cuda.synchronize()
    assert_close(o.cpu().numpy(), orc.attn_ref(qn, qg, kc_ref, vc_ref, n - T, SCALE, nkvh, n + 5, q8=False), "f16 KV")


@pytest.mark.parametrize("n,cuts", [(5000, [0, 2560, 5000]), (3000, [0, 1024, 2048, 3000])])
def test_kv_length_slices_exchanged_over_peer_memory(q27, orc, n, cuts):
    """The peer-memory exchange of the KV-length split, with all "ranks" emulated on one GPU one after
    the other (every wait finds its flag already set: kernels that wait on one another never run
    concurrently on one GPU): each rank pushes its slice into every rank's exchange buffer, each rank's
    waiting merge then gives the whole result, bit-identical to the gathered merge; three steps in a
    row exercise the step counter and the two parities of the buffers."""
    from qwen27_engine_b200 import synth
    T, nkvh = 4, 1
    nqh = nkvh * GQA
    nz = len(cuts) - 1
    rows = T * nqh
    bufs = [torch.zeros(q27.xbuf_bytes(nz, rows), dtype=torch.uint8, device="cuda") for _ in range(nz)]
    ptrs = [b.data_ptr() for b in bufs]
    for step in range(3):
        qn, qg, kf, vf = synth.decode_inputs(T, nqh, nkvh, n, start_kv=step)
        full_k, full_v = orc.fill_cache(kf, vf, n)
        slices = []
        for z in range(nz):
            lo, hi = cuts[z], cuts[z + 1]
            n_ctx = hi - lo + 3
            kc_ref, vc_ref = orc.fill_cache(kf[:, lo:hi], vf[:, lo:hi], n_ctx)
            slices.append((poisoned_cache(q27, kc_ref, nkvh, n_ctx, hi - lo), poisoned_cache(q27, vc_ref, nkvh, n_ctx, hi - lo),
                           n_ctx, lo, hi))
        parts = []
        for z, (kc, vc, n_ctx, lo, hi) in enumerate(slices):
            q27.attn_decode_partial_push(dev(qn), kc, vc, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx, lo, hi - lo, ptrs, z)
            part = torch.empty((T, nqh, 258), device="cuda")
            q27.attn_decode_partial(dev(qn), kc, vc, part, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx, lo, hi - lo)
            parts.append(part)
        gathered = torch.empty((T, nqh, AD), device="cuda")
        q27.lse_merge(torch.stack(parts).contiguous(), nz, rows * 258, rows, dev(qg), gathered)
        whole = orc.attn_ref(qn, qg, full_k, full_v, n - T, SCALE, nkvh, n)
        for z in range(nz):
            o = torch.full((T, nqh, AD), float("nan"), device="cuda")
            q27.lse_merge_wait(bufs[z], nz, rows, dev(qg), o)
            torch.cuda.synchronize()
            assert torch.equal(o, gathered), "rank %d, step %d" % (z, step)
            assert_close(o.cpu().numpy(), whole, "peer-memory merge, rank %d, step %d" % (z, step))
        assert int(bufs[0][:4].view(torch.int32).item()) == step + 1  # the step counter advanced
    assert q27.device_status() == 0


@pytest.mark.parametrize("n,cuts", [(5000, [0, 2560, 5000]), (3000, [0, 1024, 2048, 3000])])
def test_fused_exchange_equals_the_pair_of_calls(q27, orc, n, cuts):
    """q27b_attn_decode_exchange (one kernel pushes this rank's slice, waits for the others and writes the
    output) against the gathered merge. On one GPU the other ranks' slices are pushed first, with the push-only
    call, so that the rank under test finds them and never waits for a later launch; fresh buffers per rank
    under test (the other ranks' step counters do not advance here)."""
    from qwen27_engine_b200 import synth
    T, nkvh = 4, 1
    nqh = nkvh * GQA
    nz = len(cuts) - 1
    rows = T * nqh
    qn, qg, kf, vf = synth.decode_inputs(T, nqh, nkvh, n)
    slices, parts = [], []
    for z in range(nz):
        lo, hi = cuts[z], cuts[z + 1]
        n_ctx = hi - lo + 3
        kc_ref, vc_ref = orc.fill_cache(kf[:, lo:hi], vf[:, lo:hi], n_ctx)
        kc, vc = poisoned_cache(q27, kc_ref, nkvh, n_ctx, hi - lo), poisoned_cache(q27, vc_ref, nkvh, n_ctx, hi - lo)
        slices.append((kc, vc, n_ctx, lo, hi))
        part = torch.empty((T, nqh, 258), device="cuda")
        q27.attn_decode_partial(dev(qn), kc, vc, part, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx, lo, hi - lo)
        parts.append(part)
    gathered = torch.empty((T, nqh, AD), device="cuda")
    q27.lse_merge(torch.stack(parts).contiguous(), nz, rows * 258, rows, dev(qg), gathered)
    for me in range(nz):
        bufs = [torch.zeros(q27.xbuf_bytes(nz, rows), dtype=torch.uint8, device="cuda") for _ in range(nz)]
        ptrs = [b.data_ptr() for b in bufs]
        for z, (kc, vc, n_ctx, lo, hi) in enumerate(slices):
            if z != me:
                q27.attn_decode_partial_push(dev(qn), kc, vc, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx, lo, hi - lo, ptrs, z)
        torch.cuda.synchronize()
        kc, vc, n_ctx, lo, hi = slices[me]
        o = torch.full((T, nqh, AD), float("nan"), device="cuda")
        q27.attn_decode_exchange(dev(qn), dev(qg), kc, vc, o, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx, lo, hi - lo, ptrs, me)
        torch.cuda.synchronize()
        assert q27.device_status() == 0
        assert torch.equal(o, gathered), "rank %d" % me
        assert int(bufs[me][:4].view(torch.int32).item()) == 1  # its step counter advanced
        # and what it pushed is what the push-only call pushes
        other = (me + 1) % nz
        ref = [torch.zeros(q27.xbuf_bytes(nz, rows), dtype=torch.uint8, device="cuda") for _ in range(nz)]
        q27.attn_decode_partial_push(dev(qn), kc, vc, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx, lo, hi - lo,
                                     [b.data_ptr() for b in ref], me)
        torch.cuda.synchronize()
        per = rows * 258 * 8
        a0 = 256 + me * per
        assert torch.equal(bufs[other][a0:a0 + per], ref[other][a0:a0 + per])


def _tagged(parts, tag):
    """float rows -> the exchange buffer's words: {value, step tag} as int32 pairs."""
    w = torch.empty(parts.shape + (2,), dtype=torch.int32, device=parts.device)
    w[..., 0] = parts.contiguous().view(torch.int32)
    w[..., 1] = tag
    return w


def test_peer_memory_merge_reports_a_missing_slice(q27):
    """A slice that never arrives: the waiting merge gives up after its limit and says so in the status
    word (nothing hangs, nothing traps); the output is left alone."""
    nz, rows = 2, 6
    buf = torch.zeros(q27.xbuf_bytes(nz, rows), dtype=torch.uint8, device="cuda")
    words = buf[256:].view(torch.int32)[: 2 * nz * rows * 258 * 2].view(2, nz, rows, 258, 2)  # [parity][slice][row][word]
    parts = torch.randn((nz, rows, 258), device="cuda")
    parts[..., 1] = parts[..., 1].abs() + 0.5
    words[0, 0] = _tagged(parts[0], 1)  # slice 0 of step 1 is there, slice 1 is missing
    o = torch.full((rows, AD), 7.0, device="cuda")
    q27.lse_merge_wait(buf, nz, rows, None, o)
    assert q27.device_status() & 1
    assert bool((o == 7.0).all())
    # the buffer is out of step now (its CTAs left without the step's bookkeeping) and holds words of the
    # broken step: after a reset a complete step on the same buffer works again
    q27.xbuf_reset(buf)
    assert int(buf.max().item()) == 0
    words[0] = _tagged(parts, 1)  # parity 0 of step 1
    q27.lse_merge_wait(buf, nz, rows, None, o)
    want = torch.empty((rows, AD), device="cuda")
    q27.lse_merge(parts.contiguous(), nz, rows * 258, rows, None, want)
    torch.cuda.synchronize()
    assert q27.device_status() == 0
    assert torch.equal(o, want)
    assert int(buf[:4].view(torch.int32).item()) == 1  # the step counter advanced from zero


@pytest.mark.parametrize("n", [1, 64, 65, 2368, 2369, 18944, 18945])
def test_empty_chunks_leave_no_trace(q27, orc, n):
    """Chunks without a tile write no partial (37 chunks of a KV head: 64 positions fill one, 2,368 all of them; from
    18,945 on there is a tile pool): whatever an earlier call left in the workspace must not be merged."""
    T, nkvh = 1, 4
    nqh = nkvh * GQA
    nan = torch.full((T, nqh, AD), float("nan"), device="cuda")
    kc = q27.new_cache(nkvh, 20000)
    q27.attn_decode(nan, torch.zeros((T, nqh, 512), device="cuda"), kc, kc, torch.empty_like(nan), None, None,
                    pos_tensor(20000 - T), T, SCALE, nqh, nkvh, 20000)
    run_decode(q27, orc, T, nkvh, n)
    assert q27.device_status() == 0


def test_step_captured_behind_a_copy_and_another_stream(q27, orc):
    """The kernels of a step start while their predecessor drains; in a graph the predecessor may also be a copy or a
    join of two streams. The position changes between replays."""
    from qwen27_engine_b200 import synth
    T, nkvh, n_ctx = 2, 2, 4000
    nqh = nkvh * GQA
    eps, theta = 1e-6, 10000000.0 ** (-2.0 / 64)
    _, _, kf, vf = synth.decode_inputs(T, nqh, nkvh, n_ctx)
    kc_ref, vc_ref = orc.fill_cache(kf, vf, n_ctx)
    rn = lambda seed, *s: dev(synth.normal(seed, s))  # noqa: E731
    qg, k, v = rn(synth.SEED_Q, T, nqh, 512), rn(synth.SEED_K, T, nkvh, AD), rn(synth.SEED_V, T, nkvh, AD)
    w = torch.ones(AD, device="cuda")
    pos_in, pos, qg_in = pos_tensor(0), pos_tensor(0), qg.clone()
    kc, vc = dev(kc_ref), dev(vc_ref)
    qn, o = torch.empty((T, nqh, AD), device="cuda"), torch.empty((T, nqh, AD), device="cuda")

    def step(qn, o, kc, vc):
        q27.attn_prep(qg, k, v, w, w, qn, kc, vc, pos, T, eps, theta, nqh, nkvh, n_ctx)
        q27.attn_decode(qn, qg, kc, vc, o, None, None, pos, T, SCALE, nqh, nkvh, n_ctx)

    side = torch.cuda.Stream()
    step(qn, o, kc, vc)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            qg.copy_(qg_in)
        pos.copy_(pos_in)
        torch.cuda.current_stream().wait_stream(side)
        step(qn, o, kc, vc)
    for n in (100, 3000, 64):
        kc.copy_(dev(kc_ref)), vc.copy_(dev(vc_ref))
        pos_in.fill_(n - T)
        g.replay()
        torch.cuda.synchronize()
        got = o.clone()
        kc2, vc2 = dev(kc_ref), dev(vc_ref)
        o2 = torch.empty_like(o)
        step(torch.empty_like(qn), o2, kc2, vc2)
        torch.cuda.synchronize()
        assert_close(got.cpu().numpy(), o2.cpu().numpy(), "replay at n=%d" % n)
        assert torch.equal(kc, kc2) and torch.equal(vc, vc2)
    assert q27.device_status() == 0


@pytest.mark.parametrize("T", [1, 2])
def test_f16_cache_many_tiles_a_chunk(q27, orc, T):
    """Few query tokens over 13 tiles a chunk of an f16 cache: the two tile groups share an odd number of stages, and a
    fast group must not take the other's first tile for its own next one."""
    from qwen27_engine_b200 import synth
    nkvh, n = 1, 120007
    nqh, n_ctx = nkvh * GQA, n + 9
    qn, qg, kf, vf = synth.decode_inputs(T, nqh, nkvh, n)
    kc_ref, vc_ref = orc.fill_cache(kf, vf, n_ctx, q8=False)
    kc, vc = poisoned_cache(q27, kc_ref, nkvh, n_ctx, n, False), poisoned_cache(q27, vc_ref, nkvh, n_ctx, n, False)
    ref = orc.attn_ref(qn, qg, kc_ref, vc_ref, n - T, SCALE, nkvh, n_ctx, q8=False)
    for _ in range(5):
        o = torch.full((T, nqh, AD), float("nan"), device="cuda")
        q27.attn_decode(dev(qn), dev(qg), kc, vc, o, None, None, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx, False)
        torch.cuda.synchronize()
        assert_close(o.cpu().numpy(), ref, "f16 T=%d n=%d" % (T, n))
    assert q27.device_status() == 0


def _leave_nan_in_the_workspace(q27, nkvh):
    nqh = nkvh * GQA
    nan = torch.full((4, nqh, AD), float("nan"), device="cuda")
    kc = q27.new_cache(nkvh, 80000)
    q27.attn_decode(nan, torch.zeros((4, nqh, 512), device="cuda"), kc, kc, torch.empty_like(nan), None, None,
                    pos_tensor(80000 - 4), 4, SCALE, nqh, nkvh, 80000)


# 148 chunks of one KV head, 74 of two (the merge that shares a row out over CTAs): the last length with a chunk of one
# tile each, the last without a pool, and the next ones
@pytest.mark.parametrize("nkvh,n", [(1, 1), (1, 65), (1, 9472), (1, 9473), (1, 75776), (1, 75777), (2, 64), (2, 4736), (2, 4737),
                                    (2, 37888), (2, 37889), (4, 2369), (4, 18945)])
@pytest.mark.parametrize("q8", [True, False], ids=["q8", "f16"])
def test_empty_chunks_leave_no_trace_in_any_merge(q27, orc, decode_kernel, nkvh, n, q8):
    """As above for every form of the merge and for f16 caches, whose kernel cuts its chunks by a formula of its own."""
    from qwen27_engine_b200 import synth
    if not q8 and decode_kernel != 1:
        pytest.skip("f16 caches have one kernel")
    T, nqh, n_ctx = min(n, 2), nkvh * GQA, n + 9
    _leave_nan_in_the_workspace(q27, nkvh)
    qn, qg, kf, vf = synth.decode_inputs(T, nqh, nkvh, n)
    kc_ref, vc_ref = orc.fill_cache(kf, vf, n_ctx, q8=q8)
    o = torch.full((T, nqh, AD), float("nan"), device="cuda")
    q27.attn_decode(dev(qn), dev(qg), poisoned_cache(q27, kc_ref, nkvh, n_ctx, n, q8), poisoned_cache(q27, vc_ref, nkvh, n_ctx, n, q8),
                    o, None, None, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx, q8)
    torch.cuda.synchronize()
    assert_close(o.cpu().numpy(), orc.attn_ref(qn, qg, kc_ref, vc_ref, n - T, SCALE, nkvh, n_ctx, q8=q8), "nkvh=%d n=%d" % (nkvh, n))
    assert q27.device_status() == 0


@pytest.mark.parametrize("nkvh", [1, 2, 4])
@pytest.mark.parametrize("n_local", [0, 1, 65])
def test_partial_of_a_short_slice_has_no_trace(q27, orc, nkvh, n_local):
    """A slice of no, one or 65 rows of a longer sequence behind a workspace full of NaN: an empty slice is the neutral
    partial, and merged with the rest of the sequence every slice gives the whole."""
    from qwen27_engine_b200 import synth
    T, n, nqh = 2, 700, nkvh * GQA
    cut = n - n_local
    qn, qg, kf, vf = synth.decode_inputs(T, nqh, nkvh, n)
    rows, parts = T * nqh, []
    for lo, hi in ((0, cut), (cut, n)):
        n_ctx = max(hi - lo, 1) + 7
        a, b = (lo, hi) if hi > lo else (0, 1)  # rows of an empty slice's cache: anything
        kc_ref, vc_ref = orc.fill_cache(kf[:, a:b], vf[:, a:b], n_ctx)
        kc, vc = poisoned_cache(q27, kc_ref, nkvh, n_ctx, hi - lo), poisoned_cache(q27, vc_ref, nkvh, n_ctx, hi - lo)
        _leave_nan_in_the_workspace(q27, nkvh)
        part = torch.full((T, nqh, 258), float("nan"), device="cuda")
        q27.attn_decode_partial(dev(qn), kc, vc, part, pos_tensor(n - T), T, SCALE, nqh, nkvh, n_ctx, lo, hi - lo)
        parts.append(part)
    torch.cuda.synchronize()
    if n_local == 0:
        assert bool((parts[1][..., 0] == -1e30).all()) and bool((parts[1][..., 1:] == 0).all())
    o = torch.empty((T, nqh, AD), device="cuda")
    q27.lse_merge(torch.stack(parts).contiguous(), 2, rows * 258, rows, dev(qg), o)
    torch.cuda.synchronize()
    kc_ref, vc_ref = orc.fill_cache(kf, vf, n)
    assert_close(o.cpu().numpy(), orc.attn_ref(qn, qg, kc_ref, vc_ref, n - T, SCALE, nkvh, n), "slice of %d rows" % n_local)
    assert q27.device_status() == 0


def test_steps_on_two_streams_of_the_caller(q27, orc):
    """Steps issued in turn on two streams that wait for one another, neither the default one: the kernels that start
    early on one stream find what the other has written (cache rows, position, query, workspace). n stays below the tile
    pool, so the outputs are the same bits as with a synchronise behind every call."""
    from qwen27_engine_b200 import synth
    T, nkvh, n0, steps = 2, 2, 300, 12
    nqh, n_ctx = nkvh * GQA, 1000
    eps, theta = 1e-6, 10000000.0 ** (-2.0 / 64)
    _, _, kf, vf = synth.decode_inputs(T, nqh, nkvh, n_ctx)
    kc_ref, vc_ref = orc.fill_cache(kf, vf, n_ctx)
    w = torch.ones(AD, device="cuda")
    qg = [dev(synth.normal(synth.SEED_Q, (T, nqh, 512), start=i * 7919)) for i in range(steps)]
    k = [dev(synth.normal(synth.SEED_K, (T, nkvh, AD), start=i * 7919)) for i in range(steps)]
    v = [dev(synth.normal(synth.SEED_V, (T, nkvh, AD), start=i * 7919)) for i in range(steps)]

    def run(streams, sync):
        kc, vc, pos = dev(kc_ref), dev(vc_ref), pos_tensor(n0)
        qn, o = torch.empty((T, nqh, AD), device="cuda"), [torch.empty((T, nqh, AD), device="cuda") for _ in range(steps)]
        torch.cuda.synchronize()
        for i in range(steps):
            s = streams[i % 2]
            s.wait_stream(streams[(i + 1) % 2])
            with torch.cuda.stream(s):
                q27.attn_prep(qg[i], k[i], v[i], w, w, qn, kc, vc, pos, T, eps, theta, nqh, nkvh, n_ctx)
                if sync:
                    torch.cuda.synchronize()
                q27.attn_decode(qn, qg[i], kc, vc, o[i], None, None, pos, T, SCALE, nqh, nkvh, n_ctx)
                pos += T
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return o, kc, vc

    d = torch.cuda.current_stream()
    want = run((d, d), True)
    for _ in range(3):
        got = run((torch.cuda.Stream(), torch.cuda.Stream()), False)
        assert all(torch.equal(a, b) for a, b in zip(got[0], want[0]))
        assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    assert q27.device_status() == 0
