"""The whole MLA layer through fst_cuda_mla_forward (process_mla with host buffers) against
the CPU oracle on identical seeded inputs: stage by stage (the FST_MLA_TRACE stage list,
src/fst_engine.cpp:3396-3407, 3521-3532, 3685-3695, 3841-3851) and end to end."""
import numpy as np
import pytest

from fastar_b200 import mla, synth
from oracle import oracle as O
from tests.helpers import check_close, oracle_cfg

pytestmark = pytest.mark.gpu

IMPLS = [("simt", mla.IMPL_SIMT, mla.IMPL_SIMT), ("tensor", mla.IMPL_TENSOR, mla.IMPL_AUTO)]
_W = {}


def weights_for(preset, attn_norm=False):
    """Seed-0 weights of the preset at full size, as bits (GPU) and rounded fp32 (oracle).
    attn_norm: also the weight of the RMSNorm in front of the layer, N(1, 0.1^2)."""
    key = (preset, attn_norm)
    if key not in _W:
        cfg = mla.make_config(preset)
        w = synth.layer_weights_f32(cfg, 0, 0)
        if attn_norm:
            w["attn_norm"] = 1.0 + synth.normal_f32(0, "attn_norm", (cfg.hidden,), 0.1, (0,))
        _W[key] = (synth.weights_to_bits(w), synth.weights_rounded(w))
    return _W[key]


def run_layer(preset, impl, lens, q_len, causal, seed=0, steps=1, ulps=0, attn_norm=False, rope_yarn=False,
              yarn_by_layer_call=False, sizes=None):
    """`steps` consecutive layer calls (each appends q_len tokens per sequence, or q_len[b] to sequence
    b); every call is compared with the oracle, and so is the cache content afterwards.  sizes:
    configuration values other than the preset's."""
    attn_impl, gemm_impl = impl[1], impl[2]
    B = len(lens)
    q_lens = [q_len] * B if isinstance(q_len, int) else list(q_len)
    T = sum(q_lens)
    n_pages = sum((L + q * steps + 63) // 64 for L, q in zip(lens, q_lens)) + 4
    cfg = mla.make_config(preset, n_pages=n_pages, max_tokens=T, max_seqs=B, attn_impl=attn_impl,
                          gemm_impl=gemm_impl, rope_yarn=rope_yarn and not yarn_by_layer_call, **(sizes or {}))
    if sizes:
        w = synth.layer_weights_f32(cfg, 0, 0)
        bits, rounded = synth.weights_to_bits(w), synth.weights_rounded(w)
    else:
        bits, rounded = weights_for(preset, attn_norm)
    ocfg = oracle_cfg(cfg)
    ocfg.rope_yarn = int(rope_yarn)
    d = mla.dims_of(cfg)
    H = cfg.n_heads
    with mla.MlaContext(cfg) as ctx:
        ctx.set_layer_weights(0, bits)
        if yarn_by_layer_call:
            ctx.set_layer_rope(0, rope_yarn)
        seqs, caches = [], []
        for b, L in enumerate(lens):
            s = ctx.seq_alloc()
            rows = synth.to_bf16_bits(synth.cache_rows_f32(cfg, seed, b, L))
            if L:
                ctx.cache_write(0, s, 0, rows)
            seqs.append(s)
            cache = np.zeros((L + q_lens[b] * steps, d["row"]), np.float32)
            cache[:L] = synth.from_bf16_bits(rows)
            caches.append(cache)
        pos = list(lens)
        for step in range(steps):
            h = synth.to_bf16_bits(synth.hidden_f32(cfg, seed, T, (step,)))
            out = ctx.forward(0, h, seqs, pos, q_lens, causal=causal)
            stages = {k: ctx.get_stage(v) for k, v in (("qc", mla.STAGE_QC), ("kv", mla.STAGE_KV),
                                                      ("q_eff", mla.STAGE_QEFF), ("o_lat", mla.STAGE_OLAT),
                                                      ("low", mla.STAGE_LOW))}
            hf = synth.from_bf16_bits(h)
            for b in range(B):
                sl = slice(sum(q_lens[:b]), sum(q_lens[:b + 1]))
                slh = slice(sl.start * H, sl.stop * H)
                r = O.mla_forward(ocfg, rounded, hf[sl], pos[b], caches[b], causal=causal)
                # normed intermediates are O(1..8): one or two bf16 steps there exceed 2e-2
                check_close(stages["qc"][sl], r.trace["qc"], f"step {step} seq {b} qc", ulps=2)
                check_close(stages["kv"][sl], r.trace["kv"], f"step {step} seq {b} kv", ulps=2)
                check_close(stages["q_eff"][slh], r.trace["q_eff"], f"step {step} seq {b} q_eff", ulps=2)
                check_close(stages["o_lat"][slh], r.trace["o_lat"], f"step {step} seq {b} o_lat", ulps=ulps)
                check_close(stages["low"][sl], r.trace["low"], f"step {step} seq {b} low", ulps=ulps)
                check_close(out[sl], r.out, f"step {step} seq {b} out", ulps=ulps)
                # cache push: the appended rows are the kv stage rows, bit for bit, at the rows
                # the block table names
                got_rows = ctx.cache_read(0, seqs[b], pos[b], q_lens[b])
                assert np.array_equal(got_rows, stages["kv"][sl])
                pos[b] += q_lens[b]
        # the history itself is untouched
        for b, L in enumerate(lens):
            if L:
                assert np.array_equal(ctx.cache_read(0, seqs[b], 0, L),
                                      synth.to_bf16_bits(caches[b][:L]))


@pytest.mark.parametrize("impl", IMPLS, ids=[i[0] for i in IMPLS])
def test_decode_batch1_config1(impl):
    # "decode at batch 1 over a 4096-token cache"
    run_layer(mla.PRESET_BASELINE, impl, [4096], 1, False)


@pytest.mark.parametrize("impl", IMPLS, ids=[i[0] for i in IMPLS])
def test_decode_ragged_batch(impl):
    # batched decode, ragged context lengths, two consecutive steps
    run_layer(mla.PRESET_BASELINE, impl, [1030, 64, 1, 700, 0, 129, 2047, 333], 1, False, seed=1, steps=2)


@pytest.mark.parametrize("impl", IMPLS, ids=[i[0] for i in IMPLS])
def test_verify_block_causal(impl):
    # 16 query tokens per sequence, causal among themselves, appended at L .. L+15
    run_layer(mla.PRESET_BASELINE, impl, [200, 64], 16, True, seed=2)


@pytest.mark.parametrize("preset", [mla.PRESET_BASELINE, mla.PRESET_FASTAR_V4], ids=["baseline", "v4"])
@pytest.mark.parametrize("q_len,causal", [(16, True), (5, False)], ids=["verify-16", "dense-5"])
def test_blocks_of_tokens_scheduled_by_groups_of_lanes(preset, q_len, causal):
    """Calls with G >= 4 new tokens per sequence and enough pages are cut by BLOCKS (n_sm / G groups of
    G thread blocks, lane i of a group takes token i of each sequence over the group's run of page
    columns).  Lengths around page boundaries make the causal edge bite: with 255 cached rows token 0
    of a 16-token block ends in page 3 and the others reach page 4; with 1023 the block ends
    exactly at a boundary.  Against the oracle stage by stage, two consecutive calls."""
    run_layer(preset, IMPLS[1], [255, 256, 1023, 64 * 30 + 3, 700, 0, 4000], q_len, causal, seed=7, steps=2, ulps=2)


def test_block_schedule_against_the_token_schedule():
    """The same 16-token verify call under both schedules: the block schedule uses whole groups of 16
    thread blocks and leaves most tokens in one part; outputs agree to the rounding of a bf16 step
    (the parts are cut at other rows, so the fp32 sums differ in their last bits)."""
    lens, q = [3000, 1500, 2047, 900, 4100, 64], 16
    B = len(lens)
    cfg = mla.make_config(mla.PRESET_BASELINE, n_pages=sum((L + q + 63) // 64 for L in lens) + 4, max_tokens=B * q, max_seqs=B)
    bits, _ = weights_for(mla.PRESET_BASELINE)
    with mla.MlaContext(cfg) as ctx:
        ctx.set_layer_weights(0, bits)
        seqs = []
        for b, L in enumerate(lens):
            s = ctx.seq_alloc()
            ctx.cache_write(0, s, 0, synth.to_bf16_bits(synth.cache_rows_f32(cfg, 12, b, L)))
            seqs.append(s)
        h = synth.to_bf16_bits(synth.hidden_f32(cfg, 12, B * q))
        res = {}
        for key, on in (("blocks", True), ("tokens", False), ("blocks again", True)):
            ctx.set_block_schedule(on)
            out = ctx.forward(0, h, seqs, lens, [q] * B, causal=True)
            res[key] = (out.copy(), ctx.plan_info())
            for s, L in zip(seqs, lens):
                ctx.seq_truncate(s, L)
        n_sm = res["tokens"][1]["n_ctas"]
        assert res["blocks"][1]["n_ctas"] == n_sm // q * q
        assert res["blocks"][1]["kv_rows"] == res["tokens"][1]["kv_rows"] == sum(L + i + 1 for L in lens for i in range(q))
        assert res["blocks"][1]["n_partials"] < res["tokens"][1]["n_partials"]
        assert np.array_equal(res["blocks"][0], res["blocks again"][0])
        check_close(res["blocks"][0], synth.from_bf16_bits(res["tokens"][0]), "block schedule vs token schedule", ulps=1)


@pytest.mark.parametrize("impl", IMPLS, ids=[i[0] for i in IMPLS])
def test_prefill_from_empty(impl):
    # the reference's own regime: 16-token chunks from position 0 (prefill_tiled, 2957-2984)
    run_layer(mla.PRESET_BASELINE, impl, [0], 16, True, seed=3, steps=2)


@pytest.mark.parametrize("impl", IMPLS, ids=[i[0] for i in IMPLS])
def test_fastar_v4_preset(impl):
    # the live engine's form: 512-wide rows, per-head q norm, sink, inverse RoPE, grouped wo_a
    # (its outputs reach several units: the absolute bound is two bf16 steps at that magnitude)
    run_layer(mla.PRESET_FASTAR_V4, impl, [100, 0, 129], 2, True, seed=4, steps=2, ulps=2)


@pytest.mark.parametrize("impl", IMPLS, ids=[i[0] for i in IMPLS])
@pytest.mark.parametrize("preset", [mla.PRESET_BASELINE, mla.PRESET_FASTAR_V4], ids=["baseline", "v4"])
def test_attn_norm_in_front_of_the_layer(impl, preset):
    # process_layer's attention half (src/fst_engine.cpp:2687-2689): the layer call takes the rows
    # before attn_norm and applies it itself; inputs with a row scale far from 1 so that a missing
    # norm cannot pass
    run_layer(preset, impl, [300, 65], 2, True, seed=5, steps=2, ulps=2, attn_norm=True)


@pytest.mark.parametrize("preset", [mla.PRESET_BASELINE, mla.PRESET_FASTAR_V4], ids=["baseline", "v4"])
@pytest.mark.parametrize("lens,q_lens", [([70], [129]), ([200, 0], [161, 140]), ([5, 130, 0], [43, 97, 60])],
                         ids=["129", "301", "200"])
def test_ragged_prompts_of_more_than_128_tokens(preset, lens, q_lens):
    """What runs above 128 tokens, stage by stage: the persistent GEMM (batch members as the middle
    tensor-map coordinate, strided outputs, the q_pe rotation on its epilogue warps) and the 256-token tile
    with a K split, last token tiles of 1 and 45 tokens, two query rows per warp in the V4 head norm,
    attn_norm in front (V4)."""
    run_layer(preset, IMPLS[1], lens, q_lens, True, seed=8, ulps=2, attn_norm=preset == mla.PRESET_FASTAR_V4)


def test_an_odd_number_of_query_rows_in_the_head_norm():
    # 249 tokens x 33 heads: 8217 rows, two to a warp, the last warp with one
    run_layer(mla.PRESET_FASTAR_V4, ("auto", mla.IMPL_AUTO, mla.IMPL_AUTO), [20], 249, True, seed=9, ulps=2,
              sizes=dict(hidden=512, n_heads=33, q_lora=128, o_lora=128))


@pytest.mark.parametrize("impl", IMPLS, ids=[i[0] for i in IMPLS])
@pytest.mark.parametrize("preset", [mla.PRESET_BASELINE, mla.PRESET_FASTAR_V4], ids=["baseline", "v4"])
@pytest.mark.parametrize("by_call", [False, True], ids=["config", "per-layer"])
def test_yarn_rope_tables(impl, preset, by_call):
    # the YaRN tables of the compressed layers (build_rope_lut, src/fst_engine.cpp:1995-2022) on the
    # key, the query and (V4) the inverse output rotation: new rows at positions 60..67 and
    # 4090..4097, both across a page boundary; stages kv and q_eff are compared inside run_layer.
    # Far positions matter: below a few hundred the YaRN and plain angles of the slow pairs agree
    # to bf16 precision.
    run_layer(preset, impl, [60, 4090], 8, True, seed=6, ulps=2, rope_yarn=True, yarn_by_layer_call=by_call)


@pytest.mark.parametrize("preset", [mla.PRESET_BASELINE, mla.PRESET_FASTAR_V4], ids=["baseline", "v4"])
def test_a_row_does_not_depend_on_the_other_rows_of_its_call(preset):
    """Compression, norms and key rotation of 320 tokens, 16 to a call and one to a call: the same bits (up to
    16 tokens share the GEMM's token tile and K split, and every row goes through the same norm kernel)."""
    n = 16
    cfg = mla.make_config(preset, n_pages=n + 2, max_tokens=n, max_seqs=n)
    bits, _ = weights_for(preset)
    with mla.MlaContext(cfg) as ctx:
        ctx.set_layer_weights(0, bits)
        seqs = [ctx.seq_alloc() for _ in range(n)]
        for rep in range(20):
            h = synth.to_bf16_bits(synth.hidden_f32(cfg, 100 + rep, n))
            ctx.append_rows(0, h, seqs, [0] * n, [1] * n)
            qc = ctx.get_stage(mla.STAGE_QC).reshape(n, -1).copy()
            kv = ctx.get_stage(mla.STAGE_KV).reshape(n, -1).copy()
            for t, s in enumerate(seqs):
                ctx.seq_truncate(s, 0)
                ctx.append_rows(0, h[t:t + 1], [s], [0], [1])
                assert np.array_equal(ctx.get_stage(mla.STAGE_QC).reshape(-1), qc[t]), (rep, t)
                assert np.array_equal(ctx.get_stage(mla.STAGE_KV).reshape(-1), kv[t]), (rep, t)
            for s in seqs:
                ctx.seq_truncate(s, 0)


def test_yarn_and_plain_tables_differ_on_the_device():
    """A context with one plain and one YaRN layer keeps both tables per plan; the same weights and
    rows give different q_eff / kv in the rope dims only."""
    cfg = mla.make_config(mla.PRESET_FASTAR_V4, n_pages=80, max_tokens=2, max_seqs=1, n_layers=2)
    bits, _ = weights_for(mla.PRESET_FASTAR_V4)
    with mla.MlaContext(cfg) as ctx:
        ctx.set_layer_weights(0, bits)
        ctx.set_layer_weights(1, bits)
        ctx.set_layer_rope(1, True)
        s = ctx.seq_alloc()
        rows = synth.to_bf16_bits(synth.cache_rows_f32(cfg, 7, 0, 4000))
        ctx.cache_write(0, s, 0, rows)
        ctx.cache_write(1, s, 0, rows)
        h = synth.to_bf16_bits(synth.hidden_f32(cfg, 7, 2))
        kv = []
        for lid in range(2):
            ctx.forward(lid, h, [s], [4000], [2])
            kv.append(ctx.get_stage(mla.STAGE_KV).copy())
        assert np.array_equal(kv[0][:, :448], kv[1][:, :448])      # the nope part does not rotate
        assert not np.array_equal(kv[0][:, 448:], kv[1][:, 448:])  # the rope tail does, differently


def test_plan_is_kept_across_the_layers_of_a_step():
    """process_layer calls process_mla once per layer with the same seq_pos_ (src/fst_engine.cpp:2687):
    the second request for the same steps keeps the plan that is on the device, gives the same bits as
    a rebuilt plan, and anything that touches a sequence makes the next request build a new one."""
    lens, B = [130, 64, 700], 3
    cfg = mla.make_config(mla.PRESET_BASELINE, n_pages=sum((L + 66) // 64 for L in lens) + 4, max_tokens=B,
                          max_seqs=B, n_layers=2)
    bits, _ = weights_for(mla.PRESET_BASELINE)
    with mla.MlaContext(cfg) as ctx:
        for lid in range(2):
            ctx.set_layer_weights(lid, bits)
        seqs = []
        for b, L in enumerate(lens):
            s = ctx.seq_alloc()
            rows = synth.to_bf16_bits(synth.cache_rows_f32(cfg, 0, b, L))
            for lid in range(2):
                ctx.cache_write(lid, s, 0, rows)
            seqs.append(s)
        h = synth.to_bf16_bits(synth.hidden_f32(cfg, 0, B, (0,)))
        c0 = ctx.plan_counts()
        out0 = ctx.forward(0, h, seqs, lens, [1] * B)        # layer 0 of the step: builds
        out1 = ctx.forward(1, h, seqs, lens, [1] * B)        # layer 1: same steps, plan kept
        c1 = ctx.plan_counts()
        assert (c1["built"] - c0["built"], c1["reused"] - c0["reused"]) == (1, 1)
        assert np.array_equal(out0, out1)                    # same weights, same cache rows in both layers
        ctx.set_plan_reuse(False)
        out2 = ctx.forward(1, h, seqs, lens, [1] * B)        # rebuilt: same bits
        c2 = ctx.plan_counts()
        assert (c2["built"] - c1["built"], c2["reused"] - c1["reused"]) == (1, 0)
        assert np.array_equal(out1, out2)
        ctx.set_plan_reuse(True)
        # the next step (positions moved on) and a rollback both ask for a new plan
        nxt = [L + 1 for L in lens]
        ctx.forward(0, h, seqs, nxt, [1] * B)
        c3 = ctx.plan_counts()
        assert c3["built"] - c2["built"] == 1
        ctx.seq_truncate(seqs[0], lens[0])
        ctx.seq_truncate(seqs[1], lens[1])
        ctx.seq_truncate(seqs[2], lens[2])
        out3 = ctx.forward(0, h, seqs, lens, [1] * B)
        c4 = ctx.plan_counts()
        assert (c4["built"] - c3["built"], c4["reused"] - c3["reused"]) == (1, 0)
        assert np.array_equal(out0, out3)


def test_host_buffers_of_every_kind_give_the_bits_of_the_device_call():
    """fst_cuda_mla_forward with page-locked, device-addressable buffers (input copied straight from the
    caller's buffer, output rows written by the last GEMM itself), with pageable buffers of up to 32 rows
    (output written by the last GEMM to page-locked rows of the context) and of more (copied behind the
    kernels): each gives the bits of fst_cuda_mla_run_device, and the output stage is that of the last
    call, whatever kind the call before it was."""
    import torch
    n = 65
    lens = [(37 * b) % 150 for b in range(n)]
    cfg = mla.make_config(mla.PRESET_BASELINE, n_pages=sum((L + 65) // 64 for L in lens) + 4, max_tokens=n, max_seqs=n)
    bits, _ = weights_for(mla.PRESET_BASELINE)
    with mla.MlaContext(cfg) as ctx:
        ctx.set_layer_weights(0, bits)
        seqs = []
        for b, L in enumerate(lens):
            s = ctx.seq_alloc()
            if L:
                ctx.cache_write(0, s, 0, synth.to_bf16_bits(synth.cache_rows_f32(cfg, 0, b, L)))
            seqs.append(s)
        h = synth.to_bf16_bits(synth.hidden_f32(cfg, 0, n, (0,)))

        def rollback(B):
            for s, L in zip(seqs[:B], lens):
                ctx.seq_truncate(s, L)

        ref = {}
        for B in (4, 32, 33, 65):
            d_h = torch.from_numpy(h[:B].view(np.int16)).cuda()
            d_out = torch.zeros_like(d_h)
            torch.cuda.synchronize()
            ctx.plan([(s, L, 1) for s, L in zip(seqs[:B], lens)])
            ctx.run_device(0, d_h.data_ptr(), d_out.data_ptr())
            ctx.sync()
            ref[B] = d_out.cpu().numpy().view(np.uint16)
            rollback(B)
        for B in (4, 32, 33, 65, 32, 65, 4):
            out = ctx.forward(0, h[:B], seqs[:B], lens[:B], [1] * B)
            assert np.array_equal(out, ref[B]), B
            assert np.array_equal(ctx.get_stage(mla.STAGE_OUT), ref[B]), B
            rollback(B)
            if B in (32, 65):
                h_pin = torch.from_numpy(h[:B].view(np.int16).copy()).pin_memory()
                out_pin = torch.zeros_like(h_pin).pin_memory()
                call = ctx.bind_forward(0, h_pin.numpy().view(np.uint16), out_pin.numpy().view(np.uint16),
                                        np.array(seqs[:B], np.int32), np.array(lens[:B], np.int32), np.ones(B, np.int32))
                call()
                assert np.array_equal(out_pin.numpy().view(np.uint16), ref[B]), B
                assert np.array_equal(ctx.get_stage(mla.STAGE_OUT), ref[B]), B
                rollback(B)


def test_forward_with_a_window_set_on_the_context():
    """fst_cuda_mla_set_window: process_mla attends to the last `window` rows only.  Checked on the
    attention stage: the oracle's windowed attention of the Q_eff the GPU produced; the appended row
    and the other stages do not depend on the window."""
    lens, B, W = [300, 64, 1000], 3, 100
    cfg = mla.make_config(mla.PRESET_BASELINE, n_pages=sum((L + 65) // 64 for L in lens) + 4, max_tokens=B, max_seqs=B)
    bits, _ = weights_for(mla.PRESET_BASELINE)
    ocfg, H = oracle_cfg(cfg), cfg.n_heads
    with mla.MlaContext(cfg) as ctx:
        ctx.set_layer_weights(0, bits)
        seqs = []
        for b, L in enumerate(lens):
            s = ctx.seq_alloc()
            ctx.cache_write(0, s, 0, synth.to_bf16_bits(synth.cache_rows_f32(cfg, 0, b, L)))
            seqs.append(s)
        h = synth.to_bf16_bits(synth.hidden_f32(cfg, 0, B, (0,)))
        ctx.set_window(W)
        out_w = ctx.forward(0, h, seqs, lens, [1] * B)
        q_eff = synth.from_bf16_bits(ctx.get_stage(mla.STAGE_QEFF))
        o_lat = ctx.get_stage(mla.STAGE_OLAT)
        for b, (s, L) in enumerate(zip(seqs, lens)):
            cache = synth.from_bf16_bits(ctx.cache_read(0, s, 0, L + 1))
            want = O.attention_window(ocfg, q_eff[b * H:(b + 1) * H], cache, L + 1, 1, W)
            check_close(o_lat[b * H:(b + 1) * H], want, f"window, seq {b}")
        for s, L in zip(seqs, lens):
            ctx.seq_truncate(s, L)
        ctx.set_window(0)
        out_full = ctx.forward(0, h, seqs, lens, [1] * B)
        assert not np.array_equal(out_w[0], out_full[0])      # 301 rows against the last 100
        # 65 rows: the window covers them all (the split into partials differs, so not bit for bit)
        check_close(out_w[1:2], synth.from_bf16_bits(out_full[1:2]), "window covers the context")


@pytest.mark.parametrize("preset", [mla.PRESET_BASELINE, mla.PRESET_FASTAR_V4], ids=["baseline", "v4"])
@pytest.mark.parametrize("n_seqs", [45, 150], ids=["mostly-split", "mostly-whole"])
def test_tokens_finished_by_the_attention_kernel_equal_the_merge_kernel(preset, n_seqs):
    """A token whose whole context is one segment of the split-KV schedule is normalised and written
    by the attention kernel itself; with the switch off it goes through its partial and the merge
    kernel like the split ones.  Same bits either way (o_lat and the layer output), run after run,
    with the sink and the inverse RoPE of the V4 form, empty contexts included."""
    rng = np.random.default_rng(5)
    hi = 2600 if n_seqs < 100 else 400
    lens = [int(x) for x in rng.integers(40, hi, size=n_seqs - 5)] + [0, 1, 63, 64, 65]
    B, q = len(lens), 2
    cfg = mla.make_config(preset, n_pages=sum((L + q + 63) // 64 for L in lens) + 4, max_tokens=B * q, max_seqs=B)
    bits, _ = weights_for(preset)
    with mla.MlaContext(cfg) as ctx:
        ctx.set_layer_weights(0, bits)
        seqs = []
        for b, L in enumerate(lens):
            s = ctx.seq_alloc()
            if L:
                ctx.cache_write(0, s, 0, synth.to_bf16_bits(synth.cache_rows_f32(cfg, 9, b, L)))
            seqs.append(s)
        h = synth.to_bf16_bits(synth.hidden_f32(cfg, 9, B * q))
        res = {}
        for key, direct in (("direct", True), ("kernel", False), ("direct again", True)):
            ctx.set_fused_merge(direct)
            out = ctx.forward(0, h, seqs, lens, [q] * B, causal=True)
            res[key] = (out.copy(), ctx.get_stage(mla.STAGE_OLAT).copy())
            info = ctx.plan_info()
            for s, L in zip(seqs, lens):
                ctx.seq_truncate(s, L)
        # both kinds of token are present: some split over thread blocks, some whole
        assert info["n_partials"] > B * q - 5  # split tokens are present (whole ones too: the short contexts)
        a, b, c = res["direct"], res["kernel"], res["direct again"]
        assert np.array_equal(a[1], b[1]) and np.array_equal(a[0], b[0])
        assert np.array_equal(a[1], c[1]) and np.array_equal(a[0], c[0])
