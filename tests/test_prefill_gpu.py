"""Batched prefill (bt_model_prefill): tensor-core products over all rows, one-pass K/V append, causal
attention over blocks of query positions, chunked TTT update - checked stage by stage against the
oracle (oracle/staged.py) and, where the arithmetic is reproducible bit for bit, against token-by-token
decode, whose semantics it must have (the reference CLI's prefill loop, model/llama.rs:495-498)."""
import importlib

import numpy as np
import pytest

from gpu_util import load_bt, rel_err, seed_kv_caches, staged_decode_step
from oracle.staged import staged_prefill

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bt():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    return load_bt()


@pytest.fixture(scope="module")
def syn():
    return importlib.import_module("bit-ttt-engine_b200.synthetic")


@pytest.mark.parametrize("batch,n_first,n_second", [(1, 13, 7), (2, 37, 5), (5, 16, 1)])
def test_prefill_tiny_llama_then_decode_then_prefill_again(bt, oracle, syn, batch, n_first, n_second):
    cfg = syn.TINY_LLAMA_TEST  # 2 layers, hidden 256, 8 q heads / 2 kv heads (4 per group), head_dim 32
    w = syn.make_weights(cfg, seed=6000 + batch)
    gpu = syn.build_model(w, max_batch=batch)
    ref = oracle.model_from_weights(w)
    states = [ref.new_state() for _ in range(batch)]
    rng = np.random.default_rng(batch)
    staged_prefill(oracle, ref, gpu, cfg, rng.integers(0, cfg.vocab_size, size=(batch, n_first)), states)
    for _ in range(2):  # decode continues on the cache the prefill filled
        staged_decode_step(oracle, ref, gpu, cfg, rng.integers(0, cfg.vocab_size, size=batch), states)
    staged_prefill(oracle, ref, gpu, cfg, rng.integers(0, cfg.vocab_size, size=(batch, n_second)), states)  # past > 0
    assert gpu.current_pos == n_first + 2 + n_second
    assert bt.lib().bt_device_check(0) == 0


def test_prefill_first_layer_cache_equals_token_by_token(bt, oracle, syn):
    # layer 0's keys and values depend on the embeddings only, so they must be the same bytes whichever
    # way the tokens went in; the logits of the two ways agree up to the quantisers' rounding noise
    cfg = syn.TINY_LLAMA_TEST
    w = syn.make_weights(cfg, seed=6100)
    a, b = syn.build_model(w, max_batch=2), syn.build_model(w, max_batch=2)
    tokens = np.random.default_rng(3).integers(0, cfg.vocab_size, size=(2, 21))
    la, _ = a.prefill(tokens)
    for t in range(tokens.shape[1]):
        lb, _ = b.forward_one(tokens[:, t])
    for s in range(2):
        ea, eb = a.kv_cache(0).export(s, 21), b.kv_cache(0).export(s, 21)
        for x, y in zip(ea, eb):
            assert np.array_equal(x, y)
    assert rel_err(la, lb) <= 5e-2


@pytest.mark.parametrize("ttt_chunk", [1, 16])
def test_prefill_tiny_ttt(bt, oracle, syn, ttt_chunk):
    cfg = syn.BitLlamaConfig("ttt", 500, 256, 2, 4, 4, 688, inner_lr=0.01)
    w = syn.make_weights(cfg, seed=6200)
    gpu = syn.build_model(w, max_batch=3)
    ref = oracle.model_from_weights(w)
    states = [ref.new_state() for _ in range(3)]
    rng = np.random.default_rng(5)
    tokens = rng.integers(0, cfg.vocab_size, size=(3, 37))
    logits, _ = staged_prefill(oracle, ref, gpu, cfg, tokens, states, ttt_chunk=ttt_chunk)
    for li in range(cfg.num_layers):
        for s in range(3):
            assert rel_err(gpu.ttt_state(li)[s].cpu().numpy(), states[s].w[li]) <= 1e-6
    staged_decode_step(oracle, ref, gpu, cfg, rng.integers(0, cfg.vocab_size, size=3), states)
    if ttt_chunk == 1:
        # without attention every stage is reproducible: the batched prefill IS the token-by-token loop, bit for bit
        other = syn.build_model(w, max_batch=3)
        for t in range(tokens.shape[1]):
            lo, _ = other.forward_one(tokens[:, t])
        assert np.array_equal(lo, logits)
    assert bt.lib().bt_device_check(0) == 0


def test_prefill_llama8b_block_shape_long_context(bt, oracle, syn):
    # the 8B block shape (4 query heads per KV head, head_dim 128) with 2000 positions already cached:
    # every query block walks 16 tiles of keys; 1 sequence x 48 tokens and 3 sequences x 40 tokens
    cfg = syn.BitLlamaConfig("llama", 2048, 4096, 1, 32, 8, 14336, rope_theta=500000.0, max_position_embeddings=2112)
    w = syn.make_weights(cfg, seed=6300, from_latent=False)
    gpu = syn.build_model(w, max_batch=3)
    ref = oracle.model_from_weights(w)
    for batch, n in ((1, 48), (3, 40)):
        gpu.reset_kv_cache()
        states = [ref.new_state() for _ in range(batch)]
        rng = np.random.default_rng(n)
        seed_kv_caches(gpu, states, cfg, 2000, rng)
        staged_prefill(oracle, ref, gpu, cfg, rng.integers(0, cfg.vocab_size, size=(batch, n)), states)
        staged_decode_step(oracle, ref, gpu, cfg, rng.integers(0, cfg.vocab_size, size=batch), states)
    assert bt.lib().bt_device_check(0) == 0


def test_prefill_tinyllama_shape_and_chunking(bt, oracle, syn):
    # 8 query heads per KV head, head_dim 64 (two query positions per attention CTA); 2100 rows in all, so
    # the prefill is worked off in two chunks and the second one attends over the first one's cache rows
    cfg = syn.BitLlamaConfig("llama", 512, 2048, 1, 32, 4, 5632, max_position_embeddings=1100)
    w = syn.make_weights(cfg, seed=6400, from_latent=False)
    gpu = syn.build_model(w, max_batch=2)
    ref = oracle.model_from_weights(w)
    states = [ref.new_state() for _ in range(2)]
    rng = np.random.default_rng(9)
    tokens = rng.integers(0, cfg.vocab_size, size=(2, 1050))
    logits, nxt = gpu.prefill(tokens)
    assert gpu.current_pos == 1050
    # the stage-by-stage check on a short continuation (the long prefill itself would take the oracle minutes)
    for s, st in enumerate(states):
        for li in range(cfg.num_layers):
            kq, ks, vq, vs = gpu.kv_cache(li).export(s, 1050)
            st.kq[li] = [np.ascontiguousarray(kq[:, t]) for t in range(1050)]
            st.ks[li] = [np.ascontiguousarray(ks[:, t]) for t in range(1050)]
            st.vq[li] = [np.ascontiguousarray(vq[:, t]) for t in range(1050)]
            st.vs[li] = [np.ascontiguousarray(vs[:, t]) for t in range(1050)]
        st.pos = 1050
    staged_prefill(oracle, ref, gpu, cfg, rng.integers(0, cfg.vocab_size, size=(2, 9)), states)
    assert bt.lib().bt_device_check(0) == 0


def test_prefill_errors(bt, syn):
    cfg = syn.BitLlamaConfig("llama", 64, 64, 1, 2, 1, 64, max_position_embeddings=8)
    gpu = syn.build_model(syn.make_weights(cfg, seed=1))
    with pytest.raises(bt.BitTTTError) as ei:
        gpu.prefill(np.zeros((1, 9), np.int32))
    assert ei.value.status == bt.BT_ERR_SHAPE  # beyond max_position_embeddings
    with pytest.raises(bt.BitTTTError) as ei:
        gpu.prefill(np.zeros((2, 3), np.int32))
    assert ei.value.status == bt.BT_ERR_SHAPE  # more sequences than max_batch
    gpu.prefill(np.zeros((1, 8), np.int32))
    assert gpu.current_pos == 8


@pytest.mark.parametrize("hidden,heads,kv_heads,ff,batch,n", [
    (2048, 32, 4, 5632, 2, 592), (2048, 32, 4, 5632, 3, 400), (2048, 32, 4, 5632, 1, 300), (4096, 32, 8, 14336, 1, 260), (4096, 32, 8, 14336, 2, 300),
    (1024, 8, 2, 3600, 3, 670)])
def test_prefill_row_quantisers(bt, oracle, syn, hidden, heads, kv_heads, ff, batch, n):
    # RMSNorm and SiLU * up of many rows, on both sides of the row counts and lengths at which another row kernel is taken; 3600
    # inputs leave the last threads without values.  A trace wants silu(gate) * up in memory and takes it from the kernel that
    # holds rows in shared memory: logits, and the second layer's cache rows (of every token), have to be the same
    # bits; of some rows every stage is the oracle's.
    cfg = syn.BitLlamaConfig("llama", 300, hidden, 2, heads, kv_heads, ff, max_position_embeddings=n)
    w = syn.make_weights(cfg, seed=hidden + ff, from_latent=False)
    gpu, ref = syn.build_model(w, max_batch=batch), oracle.model_from_weights(w)
    tokens = np.random.default_rng(ff).integers(0, 300, (batch, n))

    def prefill():
        gpu.reset_kv_cache()
        return [gpu.prefill(tokens)[0]] + [x for li in range(2) for b in range(batch) for x in gpu.kv_cache(li).export(b, n)]

    plain = prefill()
    gpu.set_trace(True, rows=batch * n)
    for a, b in zip(plain, prefill()):
        assert np.array_equal(a, b)
    trace, rows = gpu.read_trace(batch * n), [0, 1, 131, batch * n - 1]
    for L, t in zip(ref.layers, trace):
        t = {name: x[rows] for name, x in t.items()}
        xn = oracle.rmsnorm(t["h_in"], L.norm1, ref.cfg.rms_eps)
        assert np.array_equal(t["qkv"], np.concatenate([L.q(xn), L.k(xn), L.v(xn)], axis=1))
        xn = oracle.rmsnorm(t["h_mid"], L.norm2, ref.cfg.rms_eps)
        assert rel_err(t["act"], oracle.silu_mul(L.gate(xn), L.up(xn))) <= 1e-6
        assert np.array_equal(t["h_out"], t["h_mid"] + L.down(t["act"]))
    assert bt.lib().bt_device_check(0) == 0


def attention_64(qkv, rows, heads, kv_heads, hd, past, theta):
    """softmax(q k / sqrt(hd)) v in 64 bits for one sequence: qkv [n, (heads + 2 kv_heads) hd] before the rotation (its keys
    and values unused), rows = the cache's (k bytes, k scales, v bytes, v scales) up to the last new token."""
    f = np.float64
    n, half = len(qkv), hd // 2
    inv = (1 / theta ** (np.arange(0, hd, 2, dtype=f) / hd)).astype(np.float32)
    ang = (np.arange(past, past + n, dtype=np.float32)[:, None] * inv).astype(f)[:, None]
    q = qkv[:, :heads * hd].astype(f).reshape(n, heads, hd)
    a, b = q[..., :half], q[..., half:]
    q = np.concatenate([a * np.cos(ang) - b * np.sin(ang), a * np.sin(ang) + b * np.cos(ang)], -1)
    k, v = ((x.astype(f) - 128) * s.astype(f)[..., None] for x, s in (rows[:2], rows[2:]))
    seen = np.arange(past + n)[None] <= np.arange(past, past + n)[:, None]
    out = np.empty((n, heads, hd))
    for h in range(heads):
        g = h // (heads // kv_heads)
        s = np.where(seen, q[:, h] @ k[g].T / np.sqrt(hd), -np.inf)
        p = np.exp(s - s.max(-1, keepdims=True))
        out[:, h] = p @ v[g] / p.sum(-1, keepdims=True)
    return out.reshape(n, heads * hd)


@pytest.mark.parametrize("heads,kv_heads,hd", [(4, 4, 32), (4, 2, 64), (4, 4, 96), (8, 2, 128), (8, 1, 64), (8, 4, 96), (8, 2, 96)])
@pytest.mark.parametrize("batch,past,n", [(1, 0, 2), (3, 0, 65), (2, 0, 128), (1, 127, 2), (1, 100, 29), (1, 257, 400), (31, 200, 65), (2, 150, 1)])
def test_prefill_attention_against_64_bits(bt, syn, heads, kv_heads, hd, batch, past, n):
    # partial query blocks and key tiles, tiles that end on and beside the last key, every number of heads per KV head; 31
    # sequences make 186 items and more, so that CTAs (148 at most) take several in turn; a single token (the decode kernel).  In f32 a score has a relative error of a few 2^-24 (rotation, joining of the digits, three
    # factors), which the exponential turns into |score| (< 4 here) times that, an output one of a few 2^-24 more: 5e-7
    # bounds the relative error of the whole (2-norm), about 7e-8 is what is measured.
    cfg = syn.BitLlamaConfig("llama", 300, heads * hd, 2, heads, kv_heads, 256, max_position_embeddings=past + n + 8)
    w = syn.make_weights(cfg, seed=heads + hd)
    gpu = syn.build_model(w, max_batch=batch)
    rng = np.random.default_rng(past + n)
    if past:
        gpu.prefill(rng.integers(0, 300, (batch, past)))
    gpu.set_trace(True, rows=batch * n)
    gpu.prefill(rng.integers(0, 300, (batch, n)))
    trace = gpu.read_trace(batch * n)
    for li in range(2):
        qkv, att = (np.asarray(trace[li][name]).reshape(batch, n, -1) for name in ("qkv", "att"))
        for b in range(batch):
            want = attention_64(qkv[b], gpu.kv_cache(li).export(b, past + n), heads, kv_heads, hd, past, cfg.rope_theta)
            assert np.linalg.norm(att[b] - want) <= 5e-7 * np.linalg.norm(want)
    assert bt.lib().bt_device_check(0) == 0


def rows_for_scores(rng, q, scores):
    """Key rows whose scores with the query vectors q [kv_heads, hd] (rotated) are `scores` [past], up to f32 roundings; random values."""
    kv_heads, hd = q.shape
    b = np.round(q / np.abs(q).max(-1, keepdims=True) * 127)
    scale = np.abs(scores) * np.sqrt(hd) / (q * b).sum(-1, keepdims=True)
    kq = np.where(scores[None, :, None] < 0, -b[:, None], b[:, None]) + 128
    vq = rng.integers(0, 256, kq.shape)
    return [kq.astype(np.uint8), scale.astype(np.float32), vq.astype(np.uint8), rng.uniform(0.005, 0.03, scale.shape).astype(np.float32)]


def steered_rows(rng, kind, q, past):
    at = np.arange(past)
    if kind == "growing":    # the maximum moves in every tile, as far as the last cached key
        return rows_for_scores(rng, q, at / 40)
    if kind == "falling":
        return rows_for_scores(rng, q, -at / 40)
    if kind == "creeping":   # a little more from tile to tile, value scales just below and just above a power of two
        rows = rows_for_scores(rng, q, 3 + at / 1500)
        rows[3] = rng.choice(np.nextafter(np.float32([2.0 ** -6, 2.0 ** -7, 0.011]), np.float32([0, 1, 1])), rows[3].shape)
        return rows
    if kind in ("1e6", "1e7", "1e8"):  # scores of which an f32 holds the difference to the maximum in a few bits, or hardly at all
        return rows_for_scores(rng, q, float(kind) + rng.integers(0, 4, past) + at // 128)
    if kind == "small sums":  # the largest weight belongs to a row of zeros; what is left are small negative sums
        rows = rows_for_scores(rng, q, np.where(at == 7, 40.0, np.where(at == 9, 30.3, 10.0)))
        rows[2][:], rows[3][:] = rng.integers(124, 128, rows[2].shape), 0.01
        rows[2][:, 7] = 128
        return rows
    rows = rows_for_scores(rng, q, rng.normal(0, 2, past))
    if kind == "value scales":  # powers of two up and down from tile to tile, and rows of zeros
        rows[3] = (rows[3] * 2.0 ** ((at // 128 * 7) % 24 - 12)).astype(np.float32)
        rows[2][:, at % 5 == 0], rows[3][:, at % 5 == 0] = 128, 0
    if kind == "odd scales":  # no number, negative: nothing, as for the decode kernel; the smallest, the largest that count
        rows[3][:, at % 7 == 0], rows[3][:, at % 7 == 3] = np.nan, -1.0
        rows[3][:, :128], rows[3][:, 128:] = rows[3][:, :128] * np.float32(1e-25), rows[3][:, 128:] * np.float32(1e28)
    return rows


@pytest.mark.parametrize("heads,kv_heads,hd", [(4, 4, 32), (4, 2, 64), (8, 2, 128), (8, 1, 96)])
@pytest.mark.parametrize("kind,past", [("growing", 600), ("falling", 600), ("creeping", 2000), ("1e6", 600), ("1e7", 600), ("1e8", 600), ("value scales", 1400),
                                       ("odd scales", 700), ("small sums", 140), ("random", 513), ("random", 33000)])
def test_prefill_attention_against_decode(bt, syn, heads, kv_heads, hd, kind, past):
    # Peaked, huge and unequal rows, where the reference of the weights and their bound move, and more tiles than the
    # accumulators hold (33 000 positions).  The two kernels compute the same scores and weights of the same bits and differ in the
    # order of the sums and in the maximum that a weight is relative to at first: up to 16 moves, each with three roundings
    # and an exponential good to 2^-22 at most, hence 16 * 2^-22 of the 2-norm.
    n, theta = 3, 10000.0
    cfg = syn.BitLlamaConfig("llama", 300, heads * hd, 1, heads, kv_heads, 256, max_position_embeddings=past + n, rope_theta=theta)
    gpu = syn.build_model(syn.make_weights(cfg, seed=past + hd), max_batch=1)
    rng = np.random.default_rng(past + hd)
    tokens = rng.integers(0, 300, (1, n))
    gpu.set_trace(True, rows=n)

    def prefill():
        gpu.seek(past)
        gpu.prefill(tokens)
        return gpu.read_trace(n)[0]

    qkv = prefill()["qkv"]  # of the first layer: the same whatever the cache holds
    half = hd // 2
    ang = (np.float32(past) * (1 / theta ** (np.arange(0, hd, 2) / hd)).astype(np.float32)).astype(np.float64)
    q = qkv[0, :heads * hd].astype(np.float64).reshape(kv_heads, -1, hd)[:, 0]
    q = np.concatenate([q[:, :half] * np.cos(ang) - q[:, half:] * np.sin(ang), q[:, :half] * np.sin(ang) + q[:, half:] * np.cos(ang)], -1)
    rows = steered_rows(rng, kind, q, past)
    gpu.kv_cache(0).load(0, *rows)
    trace = prefill()
    assert np.array_equal(trace["qkv"], qkv)
    cache = bt.QuantizedKVCache(past + n, 1, kv_heads, hd)
    cache.load(0, *rows)
    for i in range(n):
        pos = torch.full((1,), past + i, dtype=torch.int32, device="cuda")
        want = bt.attn_decode(cache, torch.from_numpy(qkv[i:i + 1]).cuda(), pos, heads, theta).cpu().numpy().reshape(heads, hd).astype(np.float64)
        got = trace["att"][i].reshape(heads, hd)
        assert np.isfinite(want).all()
        assert (np.linalg.norm(got - want, axis=-1) <= 16 * 2.0 ** -22 * np.linalg.norm(want, axis=-1)).all(), (kind, i)
    assert bt.lib().bt_device_check(0) == 0


@pytest.mark.parametrize("hidden,ff,batch,n", [(256, 176, 1, 65), (256, 1040, 1, 129), (1024, 4112, 3, 90), (512, 5008, 5, 199),
                                                  (4096, 14336, 1, 300), (4096, 4112, 5, 210), (2048, 5632, 8, 490)])
def test_prefill_silu_in_the_product(bt, oracle, syn, hidden, ff, batch, n):
    # silu(gate) * up in the quantiser (the first four: few row tiles, row tiles that end inside a set of 128), and leaving the
    # gate|up product itself: tiles without some of their tokens, CTA pairs and row tiles that end inside a set (the last two)
    cfg = syn.BitLlamaConfig("llama", 64, hidden, 1, hidden // 64, hidden // 128, ff, max_position_embeddings=512)
    w = syn.make_weights(cfg, seed=ff, from_latent=False)
    gpu, ref = syn.build_model(w, max_batch=batch), oracle.model_from_weights(w)
    states = [ref.new_state() for _ in range(batch)]
    staged_prefill(oracle, ref, gpu, cfg, np.random.default_rng(n).integers(0, 64, size=(batch, n)), states)
    assert bt.lib().bt_device_check(0) == 0


@pytest.mark.parametrize("arch,n", [("llama", 40), ("llama", 100), ("ttt", 100)])
def test_prefill_of_several_bases_and_a_narrow_mlp(bt, oracle, syn, arch, n):
    # the sum of a projection's bases is wider than the gate and up rows whose buffer it borrows
    cfg = syn.BitLlamaConfig(arch, 64, 512, 2, 8, 4 if arch == "llama" else 8, 64, inner_lr=0.01, max_position_embeddings=256)
    w = syn.make_weights(cfg, seed=n, n_bases=2)
    gpu, ref = syn.build_model(w, max_batch=2), oracle.model_from_weights(w)
    states = [ref.new_state() for _ in range(2)]
    staged_prefill(oracle, ref, gpu, cfg, np.random.default_rng(n).integers(0, 64, size=(2, n)), states)
    gpu.enqueue_products(2)  # (the other caller of such a buffer)
    assert bt.lib().bt_device_check(0) == 0


def test_prompts_of_more_rows_than_one_pass(bt, syn):
    # a call of more rows than the prefill works on at a time is cut by the host: the same as calls that fit one
    # pass each - bit for bit without attention, in the first layer's cache with it
    rng = np.random.default_rng(17)
    w = syn.make_weights(syn.BitLlamaConfig("ttt", 500, 128, 2, 4, 4, 256, inner_lr=0.01), seed=6600)
    tokens = rng.integers(0, 500, size=(3, 2800))
    a, b = syn.build_model(w, max_batch=3), syn.build_model(w, max_batch=3)
    la, _ = a.prefill(tokens)
    b.prefill(tokens[:, :1300])
    lb, _ = b.prefill(tokens[:, 1300:])
    assert np.array_equal(la, lb)
    cfg = syn.BitLlamaConfig("llama", 500, 256, 2, 4, 2, 512, max_position_embeddings=1000)
    w = syn.make_weights(cfg, seed=6601)
    tokens = rng.integers(0, 500, size=(9, 1000))
    a, b = syn.build_model(w, max_batch=9), syn.build_model(w, max_batch=9)
    la, _ = a.prefill(tokens)
    b.prefill(tokens[:, :400])
    lb, _ = b.prefill(tokens[:, 400:])
    for s in (0, 4, 8):
        for x, y in zip(a.kv_cache(0).export(s, 1000), b.kv_cache(0).export(s, 1000)):
            assert np.array_equal(x, y)
    # (the attention of the two cuts rounds differently, and a last bit can move an int8 value behind it by a whole step, 1/127 of
    # its row's largest: a few such steps over two layers)
    assert rel_err(la, lb) <= 5e-2
    assert bt.lib().bt_device_check(0) == 0


def test_prompt_without_memory_for_the_large_pass(bt, syn):
    # a model that cannot have the buffers of a large pass works in small ones, keeps those it has, and does not ask again
    cfg = syn.BitLlamaConfig("llama", 500, 1024, 1, 8, 2, 4096, max_position_embeddings=1700)  # 240 MB for 6800 rows, 72 for 2048
    w = syn.make_weights(cfg, seed=6602, from_latent=False)
    import torch
    free_bytes = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    tokens = np.random.default_rng(18).integers(0, 500, size=(4, 1700))
    a, b, pieces = (syn.build_model(w, max_batch=4) for _ in range(3))
    for i in range(0, 1700, 512):  # what passes of 2048 rows are
        want, _ = pieces.prefill(tokens[:, i:i + 512])
    b.prefill(tokens[:, :512])
    b.reset_kv_cache()
    torch.cuda.empty_cache()
    filler = torch.empty(free_bytes() - (150 << 20), dtype=torch.uint8, device="cuda")  # (b has the buffers of a small pass already)
    before = free_bytes()
    for _ in range(2):
        assert np.array_equal(b.prefill(tokens)[0], want)
        assert free_bytes() == before
        b.reset_kv_cache()
    assert np.array_equal(a.prefill(tokens)[0], want)
    a.reset_kv_cache()
    del filler
    torch.cuda.empty_cache()
    before = free_bytes()
    assert np.array_equal(a.prefill(tokens)[0], want) and np.array_equal(b.prefill(tokens)[0], want)
    assert free_bytes() == before
    assert bt.lib().bt_device_check(0) == 0


@pytest.mark.parametrize("n,nxt", [(257, 256), (290, 64), (40, 257)])
def test_pieces_with_and_without_silu_in_the_product(bt, oracle, syn, n, nxt):
    # the buffer of a piece that stores silu(gate) * up holds gate and up rows of a shorter piece behind it
    cfg = syn.BitLlamaConfig("llama", 64, 4096, 1, 32, 8, 14336, max_position_embeddings=600)
    w = syn.make_weights(cfg, seed=n, from_latent=False)
    gpu, ref = syn.build_model(w), oracle.model_from_weights(w)
    states, rng = [ref.new_state()], np.random.default_rng(n)
    for piece in (n, nxt):
        staged_prefill(oracle, ref, gpu, cfg, rng.integers(0, 64, size=(1, piece)), states)
    assert bt.lib().bt_device_check(0) == 0


def test_memory_of_a_long_prompt(bt, syn):
    import torch
    cfg = syn.BitLlamaConfig("llama", 64, 4096, 1, 32, 8, 4096, max_position_embeddings=4096)
    m = syn.build_model(syn.make_weights(cfg, seed=1, from_latent=False), max_batch=2)
    m.prefill(np.zeros((2, 70), np.int64))  # (kernels are loaded)
    m.reset_kv_cache()
    before = torch.cuda.mem_get_info()[0]
    m.prefill(np.zeros((2, 4096), np.int64))
    rows = 8192 * (4 * (4096 + 6144 + 4096 + 4096) + 4096 + 4 * 35)  # stream, q|k|v, attention, silu(gate) * up, int8, scales and tokens
    assert before - torch.cuda.mem_get_info()[0] <= rows + (32 << 20)
