"""Full-size checks through properties that do not need the CPU checker to finish at that size
(configurations 1-4 at the sizes BASELINE.json names): identities, constant-value invariants,
chunking invariance, determinism."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from tests.gpu_util import BF16, F32, dev, gemm_bf16, lib, ok, ptr, stream  # noqa: E402
from tests.workloads import normal_model_arrays  # noqa: E402
from tnsr_b200.nn import GptConfig  # noqa: E402
from tnsr_b200.session import B200Session  # noqa: E402


def test_config1_gemm_identity_and_row_sums_at_8192():
    """A . I = A exactly (f32 accumulation of one exact product per output) and A . ones = row sums."""
    n = 8192
    g = torch.Generator(device="cuda").manual_seed(2)
    a = (torch.rand((n, n), device="cuda", generator=g) * 2 - 1).to(torch.bfloat16)
    eye = torch.eye(n, device="cuda", dtype=torch.bfloat16)
    out = gemm_bf16(a, eye, out_dtype=BF16)
    assert torch.equal(out, a)
    del eye, out
    # integer-valued operands: every partial sum is an integer below 2^24, so any summation order gives the same f32
    ai = torch.randint(-3, 4, (n, n), device="cuda", generator=g).to(torch.bfloat16)
    ones = torch.ones((256, n), device="cuda", dtype=torch.bfloat16)
    sums = gemm_bf16(ai, ones, out_dtype=F32)
    expected = ai.float().sum(dim=1, keepdim=True).expand(n, 256)
    assert torch.equal(sums, expected)


@pytest.mark.parametrize("m", [1, 8, 64])
def test_config1_skinny_shapes_exact_on_integer_operands(m):
    n = k = 4096
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randint(-2, 3, (m, k), device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randint(-2, 3, (n, k), device="cuda", generator=g).to(torch.bfloat16)
    out = gemm_bf16(a, b, out_dtype=F32)
    assert torch.equal(out, a.float() @ b.float().T)


def test_config2_swiglu_mlp_full_size_against_f32_matmuls():
    rows, d, f = 4096, 2048, 5632
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn((rows, d), device="cuda", generator=g).to(torch.bfloat16)
    wg = (torch.randn((d, f), device="cuda", generator=g) * 0.02).to(torch.bfloat16)
    wu = (torch.randn((d, f), device="cuda", generator=g) * 0.02).to(torch.bfloat16)
    wd = (torch.randn((f, d), device="cuda", generator=g) * 0.02).to(torch.bfloat16)
    bg = torch.randn(f, device="cuda", generator=g) * 0.1
    bu = torch.randn(f, device="cuda", generator=g) * 0.1
    bd = torch.randn(d, device="cuda", generator=g) * 0.1
    packed_w = torch.empty((2 * f, d), device="cuda", dtype=torch.bfloat16)
    packed_b = torch.empty(2 * f, device="cuda", dtype=torch.float32)
    ok(lib().tnsr_b200_pack_gate_up(ptr(wg), ptr(wu), ptr(bg), ptr(bu), ptr(packed_w), ptr(packed_b), d, f, stream()))
    wdt = torch.empty((d, f), device="cuda", dtype=torch.bfloat16)
    ok(lib().tnsr_b200_transpose_bf16(ptr(wd), ptr(wdt), f, d, stream()))
    hidden = torch.empty((rows, f), device="cuda", dtype=torch.bfloat16)
    out = torch.empty((rows, d), device="cuda", dtype=torch.bfloat16)
    ok(lib().tnsr_b200_swiglu_mlp(ptr(x), ptr(packed_w), ptr(packed_b), ptr(wdt), ptr(bd), ptr(hidden), ptr(out), rows, d, f,
                                  stream()))
    torch.cuda.synchronize()
    gate = x.float() @ wg.float() + bg
    up = x.float() @ wu.float() + bu
    h_ref = (gate * torch.sigmoid(gate) * up)
    assert float((hidden.float() - h_ref).abs().max() / h_ref.abs().max()) <= 1 / 128
    ref = h_ref.to(torch.bfloat16).float() @ wd.float() + bd
    assert float((out.float() - ref).abs().max() / ref.abs().max()) <= 2e-2
    # 64 rows of the block (the first and the last 32) against the CPU checker's composition
    # down(silu(x.Wg + bg) * (x.Wu + bu)) + bd in f32, reference operation order, on the same bf16-valued operands
    from oracle import oracle
    oracle.set_threads(oracle.max_threads())
    pick = torch.cat([torch.arange(0, 32), torch.arange(rows - 32, rows)]).cuda()
    want = oracle.swiglu_mlp(x[pick].float().cpu().numpy(), wg.float().cpu().numpy(), bg.cpu().numpy(),
                             wu.float().cpu().numpy(), bu.cpu().numpy(), wd.float().cpu().numpy(), bd.cpu().numpy())
    oracle.set_threads(1)
    got = out[pick].float().cpu().numpy()
    assert np.max(np.abs(got - want)) / np.max(np.abs(want)) <= 2e-2
    # zero input rows give exactly the bias path: silu(bg) * bu . Wd + bd is the same for every row
    x.zero_()
    ok(lib().tnsr_b200_swiglu_mlp(ptr(x), ptr(packed_w), ptr(packed_b), ptr(wdt), ptr(bd), ptr(hidden), ptr(out), rows, d, f,
                                  stream()))
    torch.cuda.synchronize()
    assert torch.equal(out, out[:1].expand_as(out))


def test_config3_attention_full_size_invariants():
    """64 sessions x 16 heads x 64, capacity 4096, lengths uniform [1, 4096] (seed 4).
    V = 1 everywhere -> every output is exactly 1 (the weights sum to 1 up to bf16 rounding of 1.0);
    V = per-session constant c_b -> output c_b; permuting the sessions permutes the output rows (up to rounding)."""
    batch, heads, hd, capacity = 64, 16, 64, 4096
    d = heads * hd
    lengths = np.random.default_rng(4).integers(1, capacity + 1, size=batch).astype(np.uint32)
    g = torch.Generator(device="cuda").manual_seed(4)
    q = torch.randn((batch, d), device="cuda", generator=g).to(torch.bfloat16)
    kc = torch.randn((batch, capacity, d), device="cuda", generator=g).to(torch.bfloat16)
    vc = torch.randn((batch, capacity, d), device="cuda", generator=g).to(torch.bfloat16)
    for b, n in enumerate(lengths):          # poison what must never be read
        kc[b, int(n):] = float("nan")
        vc[b, int(n):] = float("nan")
    ws_bytes = lib().tnsr_b200_decode_attention_workspace(batch, capacity, heads, hd)
    ws = torch.zeros(ws_bytes, dtype=torch.uint8, device="cuda")

    def run(q_, k_, v_, ln_):
        out = torch.empty((batch, d), device="cuda", dtype=torch.bfloat16)
        ln_t = torch.from_numpy(np.ascontiguousarray(ln_).view(np.int32)).cuda()
        ok(lib().tnsr_b200_decode_attention(ptr(q_), ptr(k_), ptr(v_), ptr(ln_t), ptr(out), ptr(ws), ws_bytes, batch, capacity,
                                            heads, hd, stream()))
        torch.cuda.synchronize()
        assert int(ws[64:68].view(torch.int32)[0]) == 0
        return out

    base = run(q, kc, vc, lengths)
    assert bool(torch.isfinite(base.float()).all())
    assert torch.equal(base, run(q, kc, vc, lengths))                      # deterministic
    const = torch.arange(1, batch + 1, device="cuda", dtype=torch.float32).to(torch.bfloat16)
    vconst = const[:, None, None].expand(batch, capacity, d).contiguous()
    out = run(q, kc, vconst, lengths)
    assert float((out.float() - const.float()[:, None]).abs().max() / batch) <= 1 / 128
    perm = torch.randperm(batch, device="cuda", generator=g)
    permuted = run(q[perm].contiguous(), kc[perm].contiguous(), vc[perm].contiguous(), lengths[perm.cpu().numpy()])
    # the split points of the key partition move with the session order, so the merge order of a session's
    # partial results changes: equal up to rounding, not bit for bit
    assert float((permuted.float() - base[perm].float()).abs().max()) <= max(1.0, float(base.float().abs().max())) / 128
    # every session against the CPU checker's live-prefix scan (f32, reference order) on the same bf16-valued rows;
    # poisoned rows are cleared on the host copy only: the checker never reads them either, NaN * 0 aside
    from oracle import oracle
    oracle.set_threads(oracle.max_threads())
    want = np.empty((batch, d), dtype=np.float32)
    for b0 in range(0, batch, 16):
        kh = torch.nan_to_num(kc[b0:b0 + 16].float(), nan=0.0).cpu().numpy()
        vh = torch.nan_to_num(vc[b0:b0 + 16].float(), nan=0.0).cpu().numpy()
        want[b0:b0 + 16] = oracle.decode_attention(q[b0:b0 + 16].float().cpu().numpy(), kh, vh, lengths[b0:b0 + 16], heads)
    oracle.set_threads(1)
    got = base.float().cpu().numpy()
    per_session = np.max(np.abs(got - want), axis=1) / np.maximum(1.0, np.max(np.abs(want), axis=1))
    assert per_session.max() <= 1 / 128, (int(per_session.argmax()), float(per_session.max()))


def test_config4_full_width_chunking_invariance_and_determinism():
    """12 layers, d 768, 12 x 64, SwiGLU 2048, vocab 32000: prefilling 96 tokens at once or as 64 + 32 must give the
    same last-position logits to the bf16-path tolerance (2e-2 relative), the same greedy id wherever the top two
    logits are further apart than that error, and (to bf16 resolution) the same K/V rows; rerunning gives identical
    ids."""
    cfg = GptConfig(vocab_size=32000, max_sequence_length=2048, embed_dim=768, num_heads=12, feed_forward_dim=2048,
                    num_layers=12, layer_norm_epsilon=1e-5, activation="swiglu", weight_dtype="bf16")
    arrays = normal_model_arrays(cfg, seed=5, std=0.02)
    batch, prompt_len, steps = 8, 96, 24
    ids = np.random.default_rng(55).integers(0, cfg.vocab_size, size=(batch, prompt_len)).astype(np.uint32)

    def session():
        s = B200Session(cfg, batch, 160, logits_mode="last")
        for i, a in enumerate(arrays):
            s.refresh(i, a)
        return s

    prefill_logits = []

    def greedy(s, chunks):
        position, nxt = 0, None
        for c in chunks:
            logits, nxt = s.decode_full(ids[:, position:position + c], position)
            position += c
        prefill_logits.append(logits.reshape(batch, cfg.vocab_size).copy())
        out = [nxt.copy()]
        for step in range(steps):
            _, nxt = s.decode_full(nxt.reshape(batch, 1), prompt_len + step)
            out.append(nxt.copy())
        return np.stack(out)

    a = session()
    whole = greedy(a, [prompt_len])
    b = session()
    split = greedy(b, [64, 32])
    again = greedy(session(), [prompt_len])
    assert np.array_equal(whole, again)
    ka, kb = a.read_cache(0), b.read_cache(0)
    assert np.max(np.abs(ka[:, :prompt_len] - kb[:, :prompt_len])) <= np.max(np.abs(ka)) / 64
    assert np.all(ka[:, prompt_len + steps:] == 0)
    # different chunking changes which kernels (and which bf16 rounding points) produce the rows, so the logits agree
    # to the tolerance of the bf16 path and the first greedy id may differ only where the top two are that close
    lw, ls = prefill_logits[0], prefill_logits[1]
    assert np.array_equal(lw, prefill_logits[2])
    scale = float(np.max(np.abs(lw)))
    err = np.max(np.abs(lw - ls), axis=1)
    assert err.max() <= 2e-2 * scale, float(err.max() / scale)
    top2 = np.sort(lw, axis=1)[:, -2:]
    decided = (top2[:, 1] - top2[:, 0]) > 2 * err
    assert np.array_equal(whole[0][decided], split[0][decided])
    assert whole.min() >= 0 and whole.max() < cfg.vocab_size


@pytest.mark.parametrize("sessions,qkv,gate_up,down", [(32, (192, 1), (256, 1), (128, 1)), (36, (256, 1), (256, 1), (192, 1)),
                                                       (52, (256, 1), (256, 1), (256, 2))])
def test_config4_wide_tile_epilogues_agree_with_narrow_tile_epilogues(sessions, qkv, gate_up, down):
    """32 sessions x 96 tokens and more give the projections enough rows for tiles of 192 and 256 columns, whose QKV and SwiGLU epilogues run
    sixteen warps and, at 256, write through bulk tensor stores, and for pairs of CTAs; 8 sessions take narrower tiles with per-lane stores.
    The accumulation order over K does not depend on the tile shape, so the first 8 sessions must come out bit-identical: K/V rows of the
    first and the last layer and the greedy continuation."""
    cfg = GptConfig(vocab_size=32000, max_sequence_length=2048, embed_dim=768, num_heads=12, feed_forward_dim=2048,
                    num_layers=12, layer_norm_epsilon=1e-5, activation="swiglu", weight_dtype="bf16")
    arrays = normal_model_arrays(cfg, seed=5, std=0.02)
    prompt_len, steps = 96, 6
    ids = np.random.default_rng(56).integers(0, cfg.vocab_size, size=(sessions, prompt_len)).astype(np.uint32)
    columns, ctas = C.c_uint32(), C.c_uint32()
    for n, k, tile in ((3 * 768, 768, qkv), (2 * 2048, 768, gate_up), (768, 2048, down)):
        ok(lib().tnsr_b200_test_gemm_tile(sessions * prompt_len, n, k, 0, C.byref(columns), C.byref(ctas)))
        assert (columns.value, ctas.value) == tile

    def run(batch):
        s = B200Session(cfg, batch, 128, logits_mode="none")
        for i, a in enumerate(arrays):
            s.refresh(i, a)
        _, nxt = s.decode_full(ids[:batch], 0)
        out = [nxt.copy()]
        for step in range(steps):
            _, nxt = s.decode_full(nxt.reshape(batch, 1), prompt_len + step)
            out.append(nxt.copy())
        caches = [s.read_cache(i) for i in (0, 1, 2 * cfg.num_layers - 2, 2 * cfg.num_layers - 1)]
        s.close()
        return np.stack(out), caches

    wide_ids, wide = run(sessions)
    narrow_ids, narrow = run(8)
    for w, n in zip(wide, narrow):
        assert np.array_equal(w[:8, :prompt_len].view(np.uint32), n[:, :prompt_len].view(np.uint32))
    assert np.array_equal(wide_ids[:, :8], narrow_ids)


def test_config4_serving_shape_end_to_end_against_checker():
    """The configuration the benchmark times, against the CPU checker: 12 layers, d 768, 12 x 64, SwiGLU 2048, vocab
    32000, a 256-session handle, one 512-token prefill chunk (wide-tile QKV / SwiGLU epilogues with bulk tensor stores,
    the in-place residual reduce-add, four key blocks of the tcgen05 prefill attention), then nine single-token steps
    from position 512 (the first launched kernel by kernel, the rest replayed from the captured graph).  The checker
    (f32, reference operation order, bf16-rounded matrices) follows two of the 256 sessions and is fed the ids the
    library picked, so one close call does not fork the two histories.  Bar: last-position logits within 2e-2 of the
    checker's (max-abs error over max-abs value) at every step, and the same greedy id wherever the checker's top two
    logits are further apart than twice the error seen.  Mirrors tests/kv_cache.rs:29-69 (decode == full forward
    across chunk splits) at serving size."""
    from oracle import oracle
    cfg = GptConfig(vocab_size=32000, max_sequence_length=2048, embed_dim=768, num_heads=12, feed_forward_dim=2048,
                    num_layers=12, layer_norm_epsilon=1e-5, activation="swiglu", weight_dtype="bf16")
    arrays = normal_model_arrays(cfg, seed=5, std=0.02)
    batch, prefill, steps, capacity = 256, 512, 9, 528
    watched = [5, 203]                       # one session from each 128-row tile of the decode GEMMs
    ids = np.random.default_rng(57).integers(0, cfg.vocab_size, size=(batch, prefill)).astype(np.uint32)

    def run(mode):
        s = B200Session(cfg, batch, capacity, logits_mode=mode)
        for i, a in enumerate(arrays):
            s.refresh(i, a)
        logits, nxt = s.decode_full(ids, 0)
        rows = [None if logits is None else logits.reshape(batch, cfg.vocab_size)[watched].copy()]
        picks = [nxt.copy()]
        for step in range(steps):
            logits, nxt = s.decode_full(nxt.reshape(batch, 1), prefill + step)
            rows.append(None if logits is None else logits.reshape(batch, cfg.vocab_size)[watched].copy())
            picks.append(nxt.copy())
        s.close()
        return rows, np.stack(picks)

    got_logits, got_ids = run("last")
    # the benchmark's mode: no logits leave the device, the greedy id comes out of the LM-head epilogue
    _, fused_ids = run("none")
    assert np.array_equal(fused_ids, got_ids)

    oracle.set_threads(oracle.max_threads())
    ref = oracle.OracleBackend(cfg, len(watched), capacity)
    for i, a in enumerate(arrays):
        ref.refresh(i, oracle.bf16_round_np(a) if a.ndim == 2 else a)
    want = [ref.decode(ids[watched], 0).reshape(len(watched), prefill, cfg.vocab_size)[:, -1].copy()]
    for step in range(steps):
        fed = got_ids[step][watched].reshape(len(watched), 1)
        want.append(ref.decode(fed, prefill + step).reshape(len(watched), cfg.vocab_size).copy())
    oracle.set_threads(1)

    for step, (g, w) in enumerate(zip(got_logits, want)):
        assert np.all(np.isfinite(g))
        err = np.max(np.abs(g - w), axis=1)
        scale = np.max(np.abs(w), axis=1)
        assert np.all(err <= 2e-2 * scale), (step, (err / scale).tolist())
        top2 = np.sort(w, axis=1)[:, -2:]
        for j, session in enumerate(watched):
            if top2[j, 1] - top2[j, 0] > 2 * err[j]:
                assert int(got_ids[step][session]) == oracle.argmax_last(w[j]), (step, session)
