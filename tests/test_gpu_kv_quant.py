"""Quantised KV storage on the paged cache (FP8-E4M3 keys, INT4 values, float16 group scales) against the
oracle's restatement of the reference's quantiser (cpp/src/ops/kv_cache.cpp:272-399, :500-577): the stored
bytes bit for bit, the dequantised cache bit for bit, attention over it within the fp32 kernel's tolerance."""
import ctypes as C

import numpy as np
import pytest

from gpu_helpers import quant_v_offsets

pytestmark = pytest.mark.gpu


def _stored(dev, pc, b, T):
    """Bytes of sequence b, token-major: (keys (T,H,D) u8, values (T,H,D/2) u8, scales (T,H,D/32) u16)."""
    H, D, P = pc.Hkv, pc.D, pc.P
    rows = pc.max_pages * pc.B * H * P
    kq = dev.download(pc.k_pages, (rows, D), np.uint8)
    vq = dev.download(pc.v_pages, (rows // P, P * D // 2), np.uint8)       # one row per (page, kv head) block
    sc = dev.download(pc.scales, (rows, D // 32), np.uint16)
    idx = np.array([[(pc.table_host[b, t // P] * H + h) * P + t % P for h in range(H)] for t in range(T)])
    off = quant_v_offsets(P, D)                                           # where the library keeps each value byte
    vals = np.array([[vq[(pc.table_host[b, t // P] * H + h), off[t % P]] for h in range(H)] for t in range(T)])
    assert len(np.unique(off)) == off.size and off.max() == off.size - 1  # a permutation of the block's bytes
    return kq[idx], vals, sc[idx]


@pytest.mark.parametrize("D,P,T", [(128, 64, 150), (64, 16, 37), (32, 64, 5)])
def test_quantised_append_gather_match_the_oracle_bit_for_bit(D, P, T):
    from grilly_next import cabi
    from gpu_helpers import PagedCache
    from oracle import c_oracle
    dev = cabi.Device(0)
    try:
        rng = np.random.default_rng(11)
        B, H = 2, 3
        k = rng.standard_normal((B, T, H, D), dtype=np.float32)
        v = rng.standard_normal((B, T, H, D), dtype=np.float32)
        # magnitudes that exercise every branch of the encoder: an all-zero group, tiny values (code 0),
        # values below 1 after scaling (the truncated-exponent quirk), one dominant element
        k[0, 0, 0, :32] = 0.0
        k[0, 1, 1, :16] *= 1e-4
        k[1, 2, 2, 5] = 250.0
        v[0, 0, 0, :32] = 0.0
        v[1, 1, 0, 7] = -40.0
        pc = PagedCache(dev, B, H, D, T + 9, page_tokens=P, dtype=cabi.FP8_INT4, shuffle_pages=True, seed=3)
        pc.append(k[:, :T // 2], v[:, :T // 2])             # two appends: the second starts inside a page
        pc.append(k[:, T // 2:], v[:, T // 2:])
        for b in range(B):
            want = c_oracle.kv_quantize(k[b], v[b])
            got = _stored(dev, pc, b, T)
            for name, g, w in zip(("keys", "values", "scales"), got, want):
                assert np.array_equal(g, w), f"{name} of sequence {b}: {np.argwhere(g != w)[:5]}"
            gk, gv = pc.gather(b)
            wk, wv = c_oracle.kv_dequantize(*want)
            assert np.array_equal(gk.view(np.uint32), wk.view(np.uint32))
            assert np.array_equal(gv.view(np.uint32), wv.view(np.uint32))
    finally:
        dev.close()


def _dequantised(k, v):
    from oracle import c_oracle
    kd = np.stack([c_oracle.kv_dequantize(*c_oracle.kv_quantize(k[b], v[b]))[0] for b in range(k.shape[0])])
    vd = np.stack([c_oracle.kv_dequantize(*c_oracle.kv_quantize(k[b], v[b]))[1] for b in range(k.shape[0])])
    return kd, vd


def test_decode_over_the_quantised_cache():
    """The generic kernel dequantises with the reference's float32 arithmetic: 2e-4 of the oracle on the same cache."""
    from grilly_next import cabi
    from gpu_helpers import PagedCache
    from oracle import attention_oracle as orc
    dev = cabi.Device(0)
    try:
        rng = np.random.default_rng(12)
        B, Hq, Hkv, D, T = 2, 8, 2, 128, 777
        k = rng.standard_normal((B, T, Hkv, D), dtype=np.float32)
        v = rng.standard_normal((B, T, Hkv, D), dtype=np.float32)
        q = rng.standard_normal((B, 1, Hq, D), dtype=np.float32)
        pc = PagedCache(dev, B, Hkv, D, 832, dtype=cabi.FP8_INT4)
        pc.append(k, v)
        kd, vd = _dequantised(k, v)
        want = orc.gqa_decode_attention(q, kd, vd, Hq, Hkv, D)
        for splits in (1, 5):
            got = pc.decode(q, n_splits=splits, force_simt=True)
            assert np.abs(got - want).max() <= 2e-4, splits
    finally:
        dev.close()


@pytest.mark.parametrize("Hq,Hkv,lens,P", [(8, 2, (777, 64), 64), (8, 8, (130, 1), 64), (16, 2, (1000, 999), 64),
                                           (3, 1, (65, 447), 64), (32, 8, (4352, 4100), 64), (8, 2, (777, 49), 16),
                                           (16, 4, (1000, 33), 32)])
def test_tensor_core_decode_over_the_quantised_cache(Hq, Hkv, lens, P):
    """head_dim 128 with pages of 64, 32 or 16 tokens runs on the tensor-core kernel (q and P rounded to float16, the cache
    dequantised in registers): 1e-3 of the output's scale against the oracle on the same quantised cache, for unsplit,
    split and kernel-chosen launches, ragged lengths and scattered pages; and it is the kernel that ran."""
    from grilly_next import cabi
    from gpu_helpers import PagedCache
    from oracle import attention_oracle as orc
    dev = cabi.Device(0)
    try:
        rng = np.random.default_rng(Hq * 100 + Hkv)
        B, D, T = len(lens), 128, max(lens)
        k = rng.standard_normal((B, T, Hkv, D), dtype=np.float32) * rng.uniform(0.2, 3.0, (B, T, Hkv, 1)).astype(np.float32)
        v = rng.standard_normal((B, T, Hkv, D), dtype=np.float32)
        q = rng.standard_normal((B, 1, Hq, D), dtype=np.float32)
        pc = PagedCache(dev, B, Hkv, D, T + 64, page_tokens=P, dtype=cabi.FP8_INT4, shuffle_pages=True, seed=5)
        pc.append(k, v)
        cut = np.array(lens, np.int32)                      # shorten the sequences: the pages keep their tails
        dev.L.grl_memcpy_h2d(dev.h, pc.seq_lens, cut.ctypes.data_as(C.c_void_p), cut.nbytes)
        dev.sync()
        pc.lens[:] = cut
        kd, vd = _dequantised(k, v)
        want = np.concatenate([orc.gqa_decode_attention(q[b:b + 1], kd[b:b + 1, :lens[b]], vd[b:b + 1, :lens[b]], Hq, Hkv, D)
                               for b in range(B)])
        tol = 1e-3 * np.abs(want).max()
        before = dev.L.grl_launch_count()
        for splits in (1, 0, 3):
            got = pc.decode(q, n_splits=splits)
            assert np.abs(got - want).max() <= tol, (splits, np.abs(got - want).max(), tol)
        assert dev.L.grl_launch_count() - before == 3        # one launch each: the kernel merges its own splits
        simt = pc.decode(q, n_splits=2, force_simt=True)
        assert np.abs(simt - want).max() <= tol
    finally:
        dev.close()


@pytest.mark.parametrize("Hq,Hkv,lens,P,splits", [
    (8, 2, (768,), 64, 1), (8, 2, (767,), 64, 1), (4, 1, (897, 12), 32, 1), (16, 2, (2000, 1, 1985), 64, 1),       # 12 stages; the ring's 14
    (8, 8, (5000,), 16, 1), (32, 8, (9000, 8999), 64, 5), (3, 1, (16400,), 16, 17), (8, 2, (40000,), 64, 48)])     # clusters; splits apart
def test_one_cta_an_sm_decode_over_the_quantised_cache(Hq, Hkv, lens, P, splits):
    """Splits of 12 stages and more, no more CTAs than SMs: twelve compute and four producer warps a CTA.  Against the oracle on the
    same quantised cache and against the form of short splits, tolerance as for the other tensor-core cases."""
    from grilly_next import cabi
    from gpu_helpers import PagedCache
    from oracle import attention_oracle as orc
    dev = cabi.Device(0)
    try:
        rng = np.random.default_rng(sum(lens) + P)
        B, D, T = len(lens), 128, max(lens)
        k = rng.standard_normal((B, T, Hkv, D), dtype=np.float32) * rng.uniform(0.2, 3.0, (B, T, Hkv, 1)).astype(np.float32)
        v = rng.standard_normal((B, T, Hkv, D), dtype=np.float32)
        q = rng.standard_normal((B, 1, Hq, D), dtype=np.float32)
        pc = PagedCache(dev, B, Hkv, D, T + 64, page_tokens=P, dtype=cabi.FP8_INT4, shuffle_pages=True, seed=6)
        pc.append(k, v)
        cut = np.array(lens, np.int32)
        dev.L.grl_memcpy_h2d(dev.h, pc.seq_lens, cut.ctypes.data_as(C.c_void_p), cut.nbytes)
        dev.sync()
        pc.lens[:] = cut
        kd, vd = _dequantised(k, v)
        want = np.concatenate([orc.gqa_decode_attention(q[b:b + 1], kd[b:b + 1, :lens[b]], vd[b:b + 1, :lens[b]], Hq, Hkv, D)
                               for b in range(B)])
        tol = 1e-3 * np.abs(want).max()
        got = pc.decode(q, n_splits=splits)
        assert np.abs(got - want).max() <= tol
        part = pc.decode(q, n_splits=max(2, splits), partial=True)
        o, l = part[:B * Hq * D].reshape(B, 1, Hq, D), part[B * Hq * (D + 1):].reshape(B, 1, Hq, 1)
        assert np.abs(o / l - want).max() <= tol
        assert np.abs(pc.decode(q, n_splits=min(256, (T + 63) // 64 // 4)) - want).max() <= tol        # short splits
    finally:
        dev.close()


@pytest.mark.parametrize("B,Hkv,group,T,P,splits", [
    (75, 2, 4, 2560, 64, 3), (50, 3, 8, 2700, 16, 3), (75, 2, 1, 2496, 64, 1), (100, 3, 2, 2600, 64, 1)])    # 40 stages; 39; too many heads
def test_heads_just_past_the_sms_decode_in_thirds(B, Hkv, group, T, P, splits):
    """More quantised (sequence, head) pairs than SMs, two rounds of clusters of three: ragged lengths (some shorter than a third of
    the longest, one of 1), with no workspace at all where an unsplit call needs none.  Three sequences against the oracle on the same
    quantised cache, all of them against unsplit launches, tolerance as for the other tensor-core cases."""
    from grilly_next import cabi
    from gpu_helpers import PagedCache
    from oracle import attention_oracle as orc
    dev = cabi.Device(0)
    try:
        rng = np.random.default_rng(B + T)
        D, Hq = 128, Hkv * group
        k, v = rng.standard_normal((B, T, Hkv, D), dtype=np.float32), rng.standard_normal((B, T, Hkv, D), dtype=np.float32)
        q = rng.standard_normal((B, 1, Hq, D), dtype=np.float32)
        pc = PagedCache(dev, B, Hkv, D, T + 64, page_tokens=P, dtype=cabi.FP8_INT4, shuffle_pages=True, seed=7)
        pc.append(k, v)
        cut = rng.integers(1, T + 1, B).astype(np.int32)
        cut[0], cut[1], cut[2] = T, 1, T // 3
        dev.L.grl_memcpy_h2d(dev.h, pc.seq_lens, cut.ctypes.data_as(C.c_void_p), cut.nbytes)
        dev.sync()
        pc.lens[:] = cut
        kd, vd = _dequantised(k[:3], v[:3])
        want = np.concatenate([orc.gqa_decode_attention(q[b:b + 1], kd[b:b + 1, :cut[b]], vd[b:b + 1, :cut[b]], Hq, Hkv, D) for b in range(3)])
        whole = pc.decode(q, n_splits=1)
        got = pc.decode(q)
        assert pc.last_splits == splits
        tol = 1e-3 * np.abs(want).max()
        assert np.abs(got[:3] - want).max() <= tol and np.abs(whole[:3] - want).max() <= tol
        assert np.abs(got - whole).max() <= 2 * tol * max(1.0, np.abs(whole).max() / np.abs(want).max())       # tol of each side's own scale
        part = pc.decode(q, partial=True)
        o, l = part[:B * Hq * D].reshape(B, 1, Hq, D), part[B * Hq * (D + 1):].reshape(B, 1, Hq, 1)
        np.testing.assert_allclose(o / l, got, rtol=1e-5, atol=1e-6)          # the same merge; the division is fp32 on both sides
        qd, od = dev.upload(q), dev.malloc(q.nbytes)
        p = cabi.DecodeParams()
        p.kv = pc.layout()
        p.q, p.out, p.num_q_heads, p.max_seq_len = qd, od, Hq, T
        cabi.check(dev.L.grl_gqa_decode(dev.h, C.byref(p)))
        np.testing.assert_array_equal(dev.download(od, q.shape, np.float32), got)
        dev.free(qd)
        dev.free(od)
    finally:
        dev.close()


@pytest.mark.parametrize("B,Hkv,T,P,splits", [(2, 5, 41 * 8 * 64, 64, 14), (5, 8, 41 * 2 * 64 - 63, 32, 3), (2, 5, 40 * 8 * 64, 64, 8)])
def test_long_splits_that_are_no_power_of_two(B, Hkv, T, P, splits):
    """As many splits as the SMs hold where a power of two of them would be too long for clusters: ragged lengths, one of a single token
    (its other splits are empty), against the oracle on the same quantised cache, tolerance as for the other tensor-core cases."""
    from grilly_next import cabi
    from gpu_helpers import PagedCache
    from oracle import attention_oracle as orc
    dev = cabi.Device(0)
    try:
        rng = np.random.default_rng(B + T)
        D, Hq = 128, 2 * Hkv
        k, v = (rng.standard_normal((B, T, Hkv, D), dtype=np.float32) for _ in range(2))
        q = rng.standard_normal((B, 1, Hq, D), dtype=np.float32)
        pc = PagedCache(dev, B, Hkv, D, T + 64, page_tokens=P, dtype=cabi.FP8_INT4, shuffle_pages=True, seed=9)
        pc.append(k, v)
        cut = np.array([T, 1, T // 3, T - 7, 700][:B], np.int32)
        dev.L.grl_memcpy_h2d(dev.h, pc.seq_lens, cut.ctypes.data_as(C.c_void_p), cut.nbytes)
        dev.sync()
        pc.lens[:] = cut
        kd, vd = _dequantised(k, v)
        want = np.concatenate([orc.gqa_decode_attention(q[b:b + 1], kd[b:b + 1, :cut[b]], vd[b:b + 1, :cut[b]], Hq, Hkv, D) for b in range(B)])
        got = pc.decode(q)
        assert pc.last_splits == splits
        assert np.abs(got - want).max() <= 1e-3 * np.abs(want).max()
    finally:
        dev.close()


@pytest.mark.parametrize("B,Hkv,T,longest", [(2, 8, 1500, 131072), (1, 2, 50000, 131072), (20, 5, 700, 4096)])
def test_workspace_sized_at_the_longest_length_serves_shorter_ones(B, Hkv, T, longest):
    """Fewer splits are chosen at the longest length than at this one: the call takes what the workspace holds."""
    from grilly_next import cabi
    from gpu_helpers import PagedCache
    dev = cabi.Device(0)
    try:
        rng = np.random.default_rng(T)
        k, v = (rng.standard_normal((B, T, Hkv, 128), dtype=np.float32) for _ in range(2))
        q = rng.standard_normal((B, 1, Hkv, 128), dtype=np.float32)
        pc = PagedCache(dev, B, Hkv, 128, T + 64, page_tokens=64, dtype=cabi.FP8_INT4, seed=8)
        pc.append(k, v)
        want = pc.decode(q)
        splits, size, one = C.c_int(), C.c_size_t(), C.c_size_t()
        p = cabi.DecodeParams()
        p.kv = pc.layout()
        qd, od = dev.upload(q), dev.malloc(q.nbytes)
        p.q, p.out, p.num_q_heads, p.max_seq_len = qd, od, Hkv, longest
        cabi.check(dev.L.grl_decode_pick_splits(dev.h, C.byref(p), C.byref(splits)))
        assert splits.value < pc.last_splits
        cabi.check(dev.L.grl_decode_workspace_bytes(C.byref(p), splits.value, C.byref(size)))
        cabi.check(dev.L.grl_decode_workspace_bytes(C.byref(p), 1, C.byref(one)))
        ws = dev.malloc(size.value)
        p.max_seq_len, p.workspace, p.workspace_bytes = T, ws, size.value
        cabi.check(dev.L.grl_gqa_decode(dev.h, C.byref(p)))
        got = dev.download(od, q.shape, np.float32)
        assert np.abs(got - want).max() <= 1e-3 * np.abs(want).max()
        p.workspace_bytes = one.value - 4                     # less than any count needs: refused as before
        assert dev.L.grl_gqa_decode(dev.h, C.byref(p)) != 0
        for x in (qd, od, ws):
            dev.free(x)
    finally:
        dev.close()


def test_no_workspace_at_any_length_where_the_longest_needs_none():
    """100 heads: unsplit at the longest length, two splits at this one.  Without a workspace the call is unsplit here too; rows that
    leave un-normalised still need one."""
    from grilly_next import cabi
    from gpu_helpers import PagedCache
    dev = cabi.Device(0)
    try:
        rng = np.random.default_rng(15)
        B, Hkv, T = 20, 5, 700
        k, v = (rng.standard_normal((B, T, Hkv, 128), dtype=np.float32) for _ in range(2))
        q = rng.standard_normal((B, 1, Hkv, 128), dtype=np.float32)
        pc = PagedCache(dev, B, Hkv, 128, T + 64, page_tokens=64, dtype=cabi.FP8_INT4, seed=8)
        pc.append(k, v)
        pc.decode(q)
        assert pc.last_splits == 2
        want = pc.decode(q, n_splits=1)
        splits = C.c_int()
        p = cabi.DecodeParams()
        p.kv = pc.layout()
        qd, od, pd = dev.upload(q), dev.malloc(q.nbytes), dev.malloc(B * Hkv * 130 * 4)
        p.q, p.out, p.num_q_heads, p.max_seq_len = qd, od, Hkv, 4096
        cabi.check(dev.L.grl_decode_pick_splits(dev.h, C.byref(p), C.byref(splits)))
        assert splits.value == 1
        p.max_seq_len = T
        cabi.check(dev.L.grl_gqa_decode(dev.h, C.byref(p)))
        np.testing.assert_array_equal(dev.download(od, q.shape, np.float32), want)
        p.partial_out = pd
        assert dev.L.grl_gqa_decode(dev.h, C.byref(p)) != 0 and b"workspace" in dev.L.grl_last_error()
        for x in (qd, od, pd):
            dev.free(x)
    finally:
        dev.close()


def test_quantised_append_with_rope_and_queries():
    """RoPE of the new keys happens before the quantiser; the step's queries are rotated alongside."""
    from grilly_next import cabi
    from gpu_helpers import PagedCache
    from oracle import attention_oracle as orc, c_oracle
    dev = cabi.Device(0)
    try:
        rng = np.random.default_rng(13)
        B, Hq, Hkv, D, T = 1, 4, 2, 64, 40
        k = rng.standard_normal((B, T, Hkv, D), dtype=np.float32)
        v = rng.standard_normal((B, T, Hkv, D), dtype=np.float32)
        q = rng.standard_normal((B, T, Hq, D), dtype=np.float32)
        pc = PagedCache(dev, B, Hkv, D, 64, page_tokens=16, dtype=cabi.FP8_INT4)
        q_rot = pc.append(k, v, q=q, rope_mode=cabi.ROPE_INTERLEAVED)
        pos = np.arange(T)
        k_rot = orc.rope_interleaved(k.transpose(0, 2, 1, 3), pos).transpose(0, 2, 1, 3)
        np.testing.assert_allclose(q_rot, orc.rope_interleaved(q.transpose(0, 2, 1, 3), pos).transpose(0, 2, 1, 3), atol=2e-6)
        wk, wv = c_oracle.kv_dequantize(*c_oracle.kv_quantize(k_rot[0], v[0]))
        gk, gv = pc.gather(0)
        # the rotation differs in the last bit here and there, which may move a key across a code boundary
        assert np.mean(gk != wk) < 0.01 and np.abs(gk - wk).max() <= 0.13 * np.abs(wk).max()
        assert np.array_equal(gv, wv)
        assert (dev.download(pc.seq_lens, (B,), np.int32) == T).all()
    finally:
        dev.close()


@pytest.mark.parametrize("D,Hq,Hkv,n", [(128, 32, 8, 1), (128, 4, 1, 8), (128, 3, 3, 2), (64, 70, 2, 7), (32, 5, 5, 6), (32, 2, 1, 32), (256, 8, 4, 1)])
@pytest.mark.parametrize("mode", ["none", "interleaved", "half"])
def test_quantised_append_in_steps_stores_what_a_bulk_append_does(D, Hq, Hkv, n, mode):
    """A step of at most 32 (token, kv head, group) warps has a kernel of its own: the same bytes as one call with
    all the tokens, and its rotated queries to the last bit but the order of one rounding, at positions that start anywhere, and the lengths advance."""
    from grilly_next import cabi
    from gpu_helpers import PagedCache
    assert n * Hkv * (D // 32) <= 32
    dev = cabi.Device(0)
    try:
        rng = np.random.default_rng(D + n)
        B, T = 2, 3 * n + 40
        k, v = (rng.standard_normal((B, T, Hkv, D), dtype=np.float32) for _ in range(2))
        q = rng.standard_normal((B, T, Hq, D), dtype=np.float32)
        kw = {"rope_mode": {"none": cabi.ROPE_NONE, "interleaved": cabi.ROPE_INTERLEAVED, "half": cabi.ROPE_HALF}[mode]}
        off = dev.upload(np.asarray([3, 70000], np.int32))
        whole, steps = (PagedCache(dev, B, Hkv, D, T, page_tokens=16, dtype=cabi.FP8_INT4, shuffle_pages=True, seed=8) for _ in range(2))
        want_q = whole.append(k, v, q=q, pos_base=5, pos_offsets=off, **kw)
        steps.append(k[:, :40], v[:, :40], pos_base=5, pos_offsets=off, **kw)
        got_q = [steps.append(k[:, t:t + n], v[:, t:t + n], q=q[:, t:t + n], pos_base=5, pos_offsets=off, **kw) for t in range(40, T, n)]
        # x0 c - x1 s with one product fused into the subtraction, which of them is the compiler's choice in each kernel: each result is
        # within half an ulp of the unfused product and of the result, 2^-24 (|x| + |y|) <= 2^-23 (|x0| + |x1|) of the exact value
        q = np.abs(q[:, 40:])
        pair = q + {"none": 0 * q, "half": np.roll(q, D // 2, -1), "interleaved": q.reshape(*q.shape[:-1], D // 2, 2)[..., ::-1].reshape(q.shape)}[mode]
        assert (np.abs(np.concatenate(got_q, 1) - want_q[:, 40:]) <= 2.0 ** -22 * pair).all()
        for b in range(B):
            for got, want in zip(_stored(dev, steps, b, T), _stored(dev, whole, b, T)):
                assert np.array_equal(got, want)
        assert (dev.download(steps.seq_lens, (B,), np.int32) == T).all()
    finally:
        dev.close()


def test_python_ops_on_a_quantised_cache():
    """create_kv_cache(use_asymmetric_quant=True): append, kv_cache_decode (dequantised, bit for bit) and decode."""
    import grilly_core
    from oracle import attention_oracle as orc, c_oracle
    ctx = grilly_core.Device()
    rng = np.random.default_rng(14)
    Hq, Hkv, D, T = 8, 2, 64, 90
    kv = grilly_core.create_kv_cache(ctx, num_heads=Hkv, head_dim=D, compression_ratio=1, max_cache_tokens=128,
                                     use_asymmetric_quant=True, use_h2o=False, page_tokens=16)
    k = rng.standard_normal((T, Hkv, D), dtype=np.float32)
    v = rng.standard_normal((T, Hkv, D), dtype=np.float32)
    grilly_core.kv_cache_append(ctx, kv, k[:50], v[:50])
    grilly_core.kv_cache_append(ctx, kv, k[50:], v[50:])
    assert kv.current_len == T
    got = grilly_core.kv_cache_decode(ctx, kv)
    wk, wv = c_oracle.kv_dequantize(*c_oracle.kv_quantize(k, v))
    assert np.array_equal(got["keys"], wk) and np.array_equal(got["values"], wv)
    q = rng.standard_normal((1, 1, Hq, D), dtype=np.float32)
    out = grilly_core.gqa_attention(ctx, q, kv)
    want = orc.gqa_decode_attention(q, wk[None], wv[None], Hq, Hkv, D)
    assert np.abs(out - want).max() <= 2e-4
    assert abs(kv.stats()["compression_ratio"] - 8.0 / 1.5) < 1e-3     # the reference's figure: scales not counted
    with pytest.raises(RuntimeError, match="quantised"):
        grilly_core.kv_cache_compact(ctx, kv)
    grilly_core.destroy_kv_cache(ctx, kv)
