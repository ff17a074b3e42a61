"""Packed variable-length prefill attention and the dense -> compressed cache build through the C ABI
(tests/attention_prefill_varlen.rs and tests/forward_with_layer_smoke.rs:332-515 of the reference)."""
import ctypes as C

import numpy as np
import pytest

import two_tiles
from helpers import assert_close

pytestmark = pytest.mark.gpu


def run_prefill(nat, O, qh, kvh, hd, pairs, seed, sync_form=False):
    rng = np.random.default_rng(seed)
    ql = np.array([p[0] for p in pairs], np.uint32)
    kl = np.array([p[1] for p in pairs], np.uint32)
    qo = np.concatenate([[0], np.cumsum(ql)[:-1]]).astype(np.uint32)
    ko = np.concatenate([[0], np.cumsum(kl)[:-1]]).astype(np.uint32)
    q = rng.standard_normal((int(ql.sum()), qh, hd)).astype(np.float32)
    k = rng.standard_normal((int(kl.sum()), kvh, hd)).astype(np.float32)
    v = rng.standard_normal((int(kl.sum()), kvh, hd)).astype(np.float32)
    dq, dk, dv, do = nat.buf(q), nat.buf(k), nat.buf(v), nat.buf(q.nbytes)
    do.upload(np.full(q.shape, 9.0, np.float32))
    dqo, dko, dql, dkl = nat.buf(qo), nat.buf(ko), nat.buf(ql), nat.buf(kl)
    f = nat.lib.m40llm_attention_prefill_f32_gqa_varlen if sync_form else nat.lib.m40llm_attention_prefill_f32_gqa_varlen_async
    rc = f(nat.ctx, dq.ptr, dk.ptr, dv.ptr, dqo.ptr, dko.ptr, dql.ptr, dkl.ptr, len(pairs), qh, kvh, hd, do.ptr)
    assert rc == 0, rc
    nat.sync(0)
    got = do.download(np.float32, q.shape)
    exp = O.attention_prefill_varlen(q, k, v, qo, ko, ql, kl, qh, kvh, hd)
    return got, exp


@pytest.mark.parametrize("hd", [64, 128])
def test_reference_prefill_case(nat, O, hd):
    """The reference test's batch: (q_len, kv_len) = (3, 3), (2, 5), (1, 4) with 4 / 2 heads."""
    for sync_form in (False, True):
        got, exp = run_prefill(nat, O, 4, 2, hd, [(3, 3), (2, 5), (1, 4)], 11 + hd, sync_form)
        assert_close(got, exp, what=f"prefill hd {hd}")
    nat.free_all()


@pytest.mark.parametrize("qh,kvh,hd,pairs", [
    (8, 2, 64, [(64, 64), (65, 65), (1, 1), (63, 200)]),          # tile boundaries
    (32, 8, 128, [(300, 300), (17, 1000), (128, 129)]),           # Llama-3-8B heads, chunked prefill with a prefix
    (16, 2, 128, [(513, 2048)]),                                  # Qwen heads, long prefix
    (32, 4, 64, [(1000, 1000), (5, 5)]),                          # TinyLlama heads
    (4, 4, 64, [(129, 129)]),                                     # MHA
])
def test_prefill_shapes(nat, O, qh, kvh, hd, pairs):
    got, exp = run_prefill(nat, O, qh, kvh, hd, pairs, qh + hd + len(pairs))
    assert_close(got, exp, what=f"prefill {qh}/{kvh} d{hd} {pairs}")
    nat.free_all()


@pytest.mark.parametrize("qh,kvh,hd,pairs", [
    (32, 8, 128, [(700, 700), (513, 1500)]),                      # pairs of heads
    (32, 4, 64, [(1001, 1001), (640, 2000)]),
    (40, 40, 64, [(769, 800), (640, 640), (1, 50)]),              # one head per group: rows that follow one another, whole and single tiles
    (33, 11, 128, [(897, 1000), (600, 600)]),                     # three heads per group
])
def test_prefill_two_row_tiles(nat, O, qh, kvh, hd, pairs):
    """More row tiles than SMs: a CTA works on two of them."""
    got, exp = run_prefill(nat, O, qh, kvh, hd, pairs, qh + hd)
    assert_close(got, exp, what=f"prefill {qh}/{kvh} d{hd} {pairs}")
    nat.free_all()


@pytest.mark.parametrize("qh,kvh,hd,pairs", two_tiles.PACKED)
def test_prefill_of_long_prompts_two_row_tiles(nat, O, qh, kvh, hd, pairs):
    got, exp = run_prefill(nat, O, qh, kvh, hd, pairs, qh + hd)
    assert_close(got, exp, what=f"prefill {qh}/{kvh} d{hd} {pairs}")
    nat.free_all()


def test_prefill_full_length_and_last_row_equals_decode(nat, O):
    """Maximum kv length the reference admits (8192), and the last q row of a prefill equals last-token decode
    attention over the same keys and values (after their f16 rounding by the cache)."""
    qh, kvh, hd, L = 8, 2, 128, 8192
    got, exp = run_prefill(nat, O, qh, kvh, hd, [(96, L)], 5)
    assert_close(got, exp, what="prefill kv 8192")
    nat.free_all()


def test_prefill_argument_errors(nat):
    f = nat.lib.m40llm_attention_prefill_f32_gqa_varlen_async
    x = nat.buf(np.zeros(4 * 64 * 8, np.float32))
    one, two, zero, big = (nat.buf(np.array([v], np.uint32)) for v in (1, 2, 0, 9000))
    assert f(nat.ctx, None, x.ptr, x.ptr, zero.ptr, zero.ptr, one.ptr, one.ptr, 1, 4, 2, 64, x.ptr) == -1
    assert f(nat.ctx, x.ptr, x.ptr, x.ptr, zero.ptr, zero.ptr, one.ptr, one.ptr, 0, 4, 2, 64, x.ptr) == -2
    assert f(nat.ctx, x.ptr, x.ptr, x.ptr, zero.ptr, zero.ptr, one.ptr, one.ptr, 1, 3, 2, 64, x.ptr) == -3
    assert f(nat.ctx, x.ptr, x.ptr, x.ptr, zero.ptr, zero.ptr, one.ptr, one.ptr, 1, 4, 2, 32, x.ptr) == -9
    assert f(nat.ctx, x.ptr, x.ptr, x.ptr, zero.ptr, zero.ptr, two.ptr, one.ptr, 1, 4, 2, 64, x.ptr) == -8   # q_len > kv_len
    assert f(nat.ctx, x.ptr, x.ptr, x.ptr, zero.ptr, zero.ptr, zero.ptr, one.ptr, 1, 4, 2, 64, x.ptr) == -8  # q_len == 0
    assert f(nat.ctx, x.ptr, x.ptr, x.ptr, zero.ptr, zero.ptr, one.ptr, big.ptr, 1, 4, 2, 64, x.ptr) == -8   # kv_len > 8192
    nat.free_all()


def test_prefill_lengths_outside_device_memory_are_refused(nat, O):
    """An array of lengths that no kernel may read is copied, as far as that goes, and never read by a kernel: the call answers with an
    error and the context goes on. The lengths are invalid, so that a machine that can copy them refuses them too."""
    x = nat.buf(np.zeros(4 * 64 * 8, np.float32))
    one, zero = nat.buf(np.array([1], np.uint32)), nat.buf(np.array([0], np.uint32))
    host = np.zeros(4096, np.uint32)
    for at in range(3):
        for ptr in (host.ctypes.data, zero.ptr + 2):   # host memory; half a value
            lens = [zero.ptr, zero.ptr, zero.ptr]      # q_lens, kv_lens, kv_offsets: no length is valid
            lens[at] = ptr
            rc = nat.lib.m40llm_attention_prefill_f32_gqa_varlen_async(nat.ctx, x.ptr, x.ptr, x.ptr, zero.ptr, lens[2], lens[0], lens[1], 1, 4, 2,
                                                                       64, x.ptr)
            assert rc in (-7, -8), rc
            nat.sync(0)
    got, exp = run_prefill(nat, O, 4, 2, 64, [(3, 3), (2, 5)], 1)
    assert_close(got, exp)
    nat.free_all()


@pytest.mark.parametrize("kvh,hd,R,bs,L", [(2, 64, 8, 4, 21), (2, 128, 16, 8, 100), (8, 128, 512, 64, 1500), (2, 64, 32, 16, 20)])
def test_build_compressed_from_dense(nat, O, kvh, hd, R, bs, L):
    """Every slot of the compressed cache ends up as token-by-token appends would have left it: bit-exact old K, q4 V
    bytes and scales, ring rows, and lengths; then block-select attention over it matches the oracle."""
    rng = np.random.default_rng(L + hd)
    slots, max_seq = 3, L + 4
    dense = nat.kv_dense(max_seq, slots, kvh, hd)
    comp = nat.kv_compressed(max_seq, slots, kvh, hd, R, bs, 3)
    ks = rng.standard_normal((slots, L, kvh, hd)).astype(np.float16)
    vs = rng.standard_normal((slots, L, kvh, hd)).astype(np.float16)
    for s in range(slots):
        nat.kv_fill(dense, s, ks[s], vs[s])
    assert nat.lib.m40llm_kvcache_build_compressed_from_dense(nat.ctx, comp, dense, L) == 0
    old_len = max(L - R, 0)
    for s in range(slots):
        old_k, q4, sc, rk, rv = O.compressed_state_from_dense(ks[s], vs[s], L, R)
        for t in sorted({0, old_len // 2, old_len - 1} & set(range(old_len))):
            k = np.empty((kvh, hd), np.float16)
            b = np.empty((kvh, hd // 2), np.uint8)
            f = np.empty(kvh, np.float32)
            assert nat.lib.m40llm_kvcache_debug_read_old_token(nat.ctx, comp, s, t, k.ctypes.data_as(C.c_void_p),
                                                               b.ctypes.data_as(C.c_void_p), f.ctypes.data_as(C.c_void_p)) == 0
            assert np.array_equal(k.view(np.uint16), old_k[t].view(np.uint16))
            assert np.array_equal(b, q4[t]) and np.array_equal(f, sc[t])
        q = rng.standard_normal(8 * hd).astype(np.float32)
        dq, do = nat.buf(q), nat.buf(q.nbytes)
        rc = nat.lib.m40llm_attention_last_token_f32_gqa_block_select_exact_fp16_k_q4_v_old_direct_async(
            nat.ctx, comp, s, dq.ptr, 8, L, R, bs, 3, do.ptr)
        assert rc == 0, rc
        nat.sync(1)
        exp, *_ = O.attention_compressed(old_k, q4, sc, rk, rv, q, 8, L, R, bs, 3)
        assert_close(do.download(np.float32, q.shape), exp, what=f"slot {s} attention over the built cache")
    # argument errors of the reference
    assert nat.lib.m40llm_kvcache_build_compressed_from_dense(nat.ctx, dense, dense, L) == -2
    assert nat.lib.m40llm_kvcache_build_compressed_from_dense(nat.ctx, comp, dense, max_seq + 1) == -4
    other = nat.kv_dense(max_seq, slots, kvh + 1, hd)
    assert nat.lib.m40llm_kvcache_build_compressed_from_dense(nat.ctx, comp, other, L) == -3
    for kv in (dense, comp, other):
        nat.lib.m40llm_kvcache_destroy(kv)
    nat.free_all()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("pos,rows,scale", [(0, 65, 1.0), (33, 100, 1.0), (0, 128, 6.0), (127, 129, 6.0), (0, 700, 6.0), (900, 257, 1.0),
                                            (895, 65, 1.0), (1033, 100, 6.0), (896, 128, 1.0), (1023, 129, 6.0), (1151, 1, 1.0)])
def test_step_rows_over_cache(nat, pkg, hd, pos, rows, scale):
    """Prompt attention over the cache at the edges of its 128 x 128 tiles; with scale 6 a row's maximum grows past its reference
    from tile to tile. Probabilities are f16: an output is off by at most 2^-11 of the largest value."""
    N = pkg.native
    rng = np.random.default_rng(hd + rows)
    qh, kvh, L = 8, 2, pos + rows
    kv = nat.kv_dense(L + 7, 4, kvh, hd)
    K, V = (rng.standard_normal((L, kvh, hd)).astype(np.float16) for _ in range(2))
    nat.kv_fill(kv, 3, K, V)
    q = (scale * rng.standard_normal((rows, qh, hd))).astype(np.float32)
    dq, do, ds = nat.buf(q), nat.buf(q.nbytes), nat.buf(np.array([0, rows, 1, pos], np.uint32))
    r = N.StepRows(rows=rows, segments=1, max_segment_rows=rows, max_len=L, slot_mul=2, slot_add=1, seg=ds.ptr)
    for _ in range(3):
        do.upload(np.full(q.shape, 9.0, np.float32))
        assert nat.lib.m40llm_attention_step_rows_async(nat.ctx, kv, dq.ptr, qh, C.byref(r), do.ptr) == 0
        nat.sync(1)
        got = do.download(np.float32, q.shape)
        for h in range(qh):
            s = q[:, h].astype(np.float64) @ K[:, h // 4].astype(np.float64).T / np.sqrt(hd)
            s[np.arange(L)[None, :] > (pos + np.arange(rows))[:, None]] = -np.inf
            p = np.exp(s - s.max(1, keepdims=True))
            want = (p / p.sum(1, keepdims=True)) @ V[:, h // 4].astype(np.float64)
            assert np.abs(got[:, h] - want).max() <= 2.0 ** -11 * float(np.abs(V).max()) + 1e-4
    nat.lib.m40llm_kvcache_destroy(kv)
    nat.free_all()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("pos,rows", [(0, 700), (1000, 129)])
@pytest.mark.parametrize("scale", [1.0, 2.0, 4.0, 8.0])
def test_prompt_forms_are_equally_exact(nat, pkg, hd, pos, rows, scale):
    """Flat to peaked scores: the tcgen05 form rounds weights to f16 relative to the running maximum as the mma.sync form does (which
    serves queries that lie on 8 bytes only), so their errors are alike; a tenth is left for their different tiles."""
    rng = np.random.default_rng(hd + rows)
    qh, kvh, L = 8, 2, pos + rows
    kv = nat.kv_dense(L, 1, kvh, hd)
    K, V = (rng.standard_normal((L, kvh, hd)).astype(np.float16) for _ in range(2))
    nat.kv_fill(kv, 0, K, V)
    q = (scale * rng.standard_normal((rows, qh, hd))).astype(np.float32)
    want = np.empty(q.shape)
    for h in range(qh):
        s = q[:, h].astype(np.float64) @ K[:, h // 4].astype(np.float64).T / np.sqrt(hd)
        s[np.arange(L)[None, :] > (pos + np.arange(rows))[:, None]] = -np.inf
        p = np.exp(s - s.max(1, keepdims=True))
        want[:, h] = (p / p.sum(1, keepdims=True)) @ V[:, h // 4].astype(np.float64)
    ds, do, error = nat.buf(np.array([0, rows, 0, pos], np.uint32)), nat.buf(q.nbytes), []
    r = pkg.native.StepRows(rows=rows, segments=1, max_segment_rows=rows, max_len=L, slot_mul=1, slot_add=0, seg=ds.ptr)
    for shift in (0, 2):
        dq = nat.buf(np.concatenate([np.zeros(shift, np.float32), q.ravel()]))
        assert nat.lib.m40llm_attention_step_rows_async(nat.ctx, kv, dq.ptr + 4 * shift, qh, C.byref(r), do.ptr) == 0
        nat.sync(1)
        error.append(np.linalg.norm(do.download(np.float32, q.shape) - want) / np.linalg.norm(want))
    assert error[0] <= 1.1 * error[1] and error[1] <= 2.0 ** -11, error
    nat.lib.m40llm_kvcache_destroy(kv)
    nat.free_all()


def poisoned(rng, L, kvh, hd, at):
    """Values, and the same with infinities and a NaN at tokens at .. at + 5 of head 0; (token, dimension, what a row that sees it gets)."""
    clean = rng.standard_normal((L, kvh, hd)).astype(np.float16)
    bad, seen = clean.copy(), []
    for token, d, value, then in ((at, 3, np.inf, np.inf), (at + 1, hd - 1, -np.inf, -np.inf), (at + 2, 10, np.nan, np.nan), (at + 5, 3, -np.inf, np.nan)):
        bad[token, 0, d] = value
        seen.append((token, d, then))
    return clean, bad, seen


def check_poisoned(got, plain, seen, pos, group):
    """Untouched dimensions keep every bit; the touched ones are computed again for rows before the token, with weights that are not
    rounded to f16 (2^-11 of a value, the largest of which is about 4)."""
    want, touched = plain.copy(), sorted({d for _, d, _ in seen})
    for token, d, then in seen:
        want[max(token - pos, 0):, :group, d] = then
    finite = np.isfinite(want)
    assert np.array_equal(got[~finite], want[~finite], equal_nan=True)
    assert np.abs(got[finite] - want[finite]).max() <= 4 * 2.0 ** -11
    untouched = np.ones(want.shape, bool)
    untouched[:, :group, touched] = False
    assert np.array_equal(got[untouched], want[untouched])


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("pos,rows,at", [(0, 40, 17), (70, 50, 100), (0, 65, 30), (0, 200, 100), (30, 300, 250), (200, 129, 305),
                                         (640, 65, 650), (768, 128, 800), (700, 129, 805)])
def test_values_that_are_not_finite_stay_with_the_rows_that_see_them(nat, pkg, hd, pos, rows, at):
    """A token whose value overflowed f16 changes the rows from it on and no earlier one; keys and values behind a sequence's last
    token and of the neighbouring sequences may be anything."""
    rng = np.random.default_rng(rows)
    qh, kvh, L = 8, 2, pos + rows
    K = rng.standard_normal((L, kvh, hd)).astype(np.float16)
    clean, bad, seen = poisoned(rng, L, kvh, hd, at)
    q = rng.standard_normal((rows, qh, hd)).astype(np.float32)
    dq, do, ds = nat.buf(q), nat.buf(q.nbytes), nat.buf(np.array([0, rows, 1, pos], np.uint32))
    r = pkg.native.StepRows(rows=rows, segments=1, max_segment_rows=rows, max_len=L, slot_mul=1, slot_add=0, seg=ds.ptr)
    out = []
    for values, around in ((clean, 0.0), (clean, np.nan), (bad, np.inf)):
        kv = nat.kv_dense(L + 150, 3, kvh, hd)
        junk = np.full((L + 150, kvh, hd), around, np.float16)
        for slot in range(3):
            nat.kv_fill(kv, slot, junk, junk)
        nat.kv_fill(kv, 1, K, values)
        assert nat.lib.m40llm_attention_step_rows_async(nat.ctx, kv, dq.ptr, qh, C.byref(r), do.ptr) == 0
        nat.sync(1)
        out.append(do.download(np.float32, q.shape))
        nat.lib.m40llm_kvcache_destroy(kv)
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])
    check_poisoned(out[2], out[0], seen, pos, qh // kvh)
    nat.free_all()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("pos,rows", [(20, 50), (0, 64), (100, 200)])
def test_packed_values_beyond_f16_stay_with_the_rows_that_see_them(nat, hd, pos, rows):
    rng = np.random.default_rng(rows + hd)
    qh, kvh, lens = 4, 2, (rows, 30)
    kv_lens, at = (pos + rows, 30), pos + rows // 2
    q = rng.standard_normal((sum(lens), qh, hd)).astype(np.float32)
    k = rng.standard_normal((sum(kv_lens), kvh, hd)).astype(np.float32)
    clean, bad, seen = poisoned(rng, sum(kv_lens), kvh, hd, at)
    offsets = [nat.buf(np.array(x, np.uint32)).ptr for x in ((0, rows), (0, kv_lens[0]), lens, kv_lens)]
    out = []
    for v in (clean, np.where(np.isinf(bad), np.sign(bad) * np.float32(1e6), bad)):
        do = nat.buf(q.nbytes)
        rc = nat.lib.m40llm_attention_prefill_f32_gqa_varlen(nat.ctx, nat.buf(q).ptr, nat.buf(k).ptr, nat.buf(v.astype(np.float32)).ptr, *offsets, 2,
                                                             qh, kvh, hd, do.ptr)
        assert rc == 0, rc
        out.append(do.download(np.float32, q.shape))
    assert np.array_equal(out[1][rows:], out[0][rows:])
    check_poisoned(out[1][:rows], out[0][:rows], seen, pos, qh // kvh)
    nat.free_all()


def over_cache(nat, pkg, kv, slot, q, pos, shift=0):
    """Rows over a cache's slot; with `shift` 2 the queries lie on 8 bytes only, which the mma.sync kernel serves."""
    rows, qh, _ = q.shape
    dq, do = nat.buf(np.concatenate([np.zeros(shift, np.float32), q.ravel()])), nat.buf(np.full(q.shape, 9.0, np.float32))
    r = pkg.native.StepRows(rows=rows, segments=1, max_segment_rows=rows, max_len=pos + rows, slot_mul=1, slot_add=0,
                            seg=nat.buf(np.array([0, rows, slot, pos], np.uint32)).ptr)
    assert nat.lib.m40llm_attention_step_rows_async(nat.ctx, kv, dq.ptr + 4 * shift, qh, C.byref(r), do.ptr) == 0
    nat.sync(1)
    return do.download(np.float32, q.shape)


@pytest.mark.parametrize("qh,kvh,hd,pos,rows", two_tiles.CACHED)
@pytest.mark.parametrize("scale", [1.0, 6.0])
def test_two_row_tiles_over_cache(nat, pkg, qh, kvh, hd, pos, rows, scale):
    """As test_step_rows_over_cache and test_prompt_forms_are_equally_exact, with two row tiles per CTA."""
    rng = np.random.default_rng(hd + rows)
    L = pos + rows
    kv = nat.kv_dense(L + 7, 2, kvh, hd)
    K, V = (rng.standard_normal((L, kvh, hd)).astype(np.float16) for _ in range(2))
    nat.kv_fill(kv, 1, K, V)
    q = (scale * rng.standard_normal((rows, qh, hd))).astype(np.float32)
    want = np.empty(q.shape)
    unseen = np.arange(L)[None, :] > (pos + np.arange(rows))[:, None]
    for h in range(qh):
        s = q[:, h].astype(np.float64) @ K[:, h // (qh // kvh)].astype(np.float64).T / np.sqrt(hd)
        s[unseen] = -np.inf
        p = np.exp(s - s.max(1, keepdims=True))
        want[:, h] = (p / p.sum(1, keepdims=True)) @ V[:, h // (qh // kvh)].astype(np.float64)
    two, plain = (over_cache(nat, pkg, kv, 1, q, pos, shift) for shift in (0, 2))
    assert np.abs(two - want).max() <= 2.0 ** -11 * float(np.abs(V).max()) + 1e-4
    error = [np.linalg.norm(x - want) / np.linalg.norm(want) for x in (two, plain)]
    assert error[0] <= 1.1 * error[1] and error[1] <= 2.0 ** -11, error
    nat.lib.m40llm_kvcache_destroy(kv)
    nat.free_all()


@pytest.mark.parametrize("qh,kvh,hd,pos,rows", two_tiles.CACHED)
@pytest.mark.parametrize("at", [3, 1000, 1290])
def test_two_row_tiles_keep_values_that_are_not_finite_with_the_rows_that_see_them(nat, pkg, qh, kvh, hd, pos, rows, at):
    """Tokens in the first, a middle and one of the last tiles: where a CTA's tiles are rows that follow one another, the first of them walks
    keys that only the second one sees."""
    rng = np.random.default_rng(rows + at)
    L = pos + rows
    K = rng.standard_normal((L, kvh, hd)).astype(np.float16)
    clean, bad, seen = poisoned(rng, L, kvh, hd, pos + at)
    q = rng.standard_normal((rows, qh, hd)).astype(np.float32)
    out = []
    for values, around in ((clean, 0.0), (clean, np.nan), (bad, np.inf)):
        kv = nat.kv_dense(L + 150, 3, kvh, hd)
        junk = np.full((L + 150, kvh, hd), around, np.float16)
        for slot in range(3):
            nat.kv_fill(kv, slot, junk, junk)
        nat.kv_fill(kv, 1, K, values)
        out.append(over_cache(nat, pkg, kv, 1, q, pos))
        nat.lib.m40llm_kvcache_destroy(kv)
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])
    check_poisoned(out[2], out[0], seen, pos, qh // kvh)
    nat.free_all()


def test_step_rows_leaves_to_the_decode_form_what_is_its(nat, pkg):
    """With the segments on the host: few rows over a long context, groups whose decode kernel keeps the weights in f32, and rows that
    do not fit the cache are handed back before anything is written; a compressed cache is refused."""
    def call(kv, hd, qh, segs):
        rows = sum(n for _, n, _ in segs)
        flat = np.array([x for i, (s, n, p) in enumerate(segs) for x in (sum(m for _, m, _ in segs[:i]), n, s, p)], np.uint32)
        q, out = nat.buf(np.ones((rows, qh, hd), np.float32)), nat.buf(np.full((rows, qh, hd), 9.0, np.float32))
        r = pkg.native.StepRows(rows=rows, segments=len(segs), max_segment_rows=max(n for _, n, _ in segs), max_len=max(n + p for _, n, p in segs),
                                slot_mul=1, slot_add=0, seg=nat.buf(flat).ptr, seg_host=flat.ctypes.data)
        rc = nat.lib.m40llm_attention_step_rows_async(nat.ctx, kv, q.ptr, qh, C.byref(r), out.ptr)
        nat.sync(1)
        return rc, bool((out.download(np.float32, (rows, qh, hd)) == 9.0).all())

    kv = nat.kv_dense(8300, 2, 4, 64)
    assert call(kv, 64, 32, [(0, 256, 300)]) == (0, False) and call(kv, 64, 32, [(0, 16, 0), (1, 40, 60)]) == (0, False)
    assert call(kv, 64, 32, [(1, 16, 8000)]) == (1, True)
    assert call(kv, 64, 32, [(1, 256, 8045)]) == (1, True)
    assert call(kv, 64, 32, [(0, 64, 0), (2, 64, 0)]) == (1, True)
    wide = nat.kv_dense(600, 1, 1, 64)
    assert call(wide, 64, 16, [(0, 256, 0)]) == (0, False) and call(wide, 64, 32, [(0, 256, 0)]) == (1, True)
    compressed = nat.kv_compressed(600, 1, 4, 64, 64, 16, 4)
    assert call(compressed, 64, 32, [(0, 256, 0)]) == (pkg.native.ERR_UNSUPPORTED, True)
    st = np.zeros(1, np.uint32)
    assert nat.lib.m40llm_context_take_device_status(nat.ctx, st.ctypes.data) == 0 and st[0] == 0
    for c in (kv, wide, compressed):
        nat.lib.m40llm_kvcache_destroy(c)
    nat.free_all()
