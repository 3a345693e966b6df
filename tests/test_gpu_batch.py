"""GPU parity of decode for more than 8 streams at once (the batched decode the reference lacks): one row per stream
through the tensor-core GEMM path, every weight format and model version, against the CPU oracle run stream by
stream.  fp16 models created for such batches keep W^T copies, quantised models a row-major copy of their packed
codes (expanded inside the GEMM); their prompts use the same path."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ABS_TOL, REL_TOL = 1e-2, 1e-3
STR = {"fp16": ("cuda fp16", "fp16"), "int8": ("cuda int8", "fp32"), "int4": ("cuda int4", "fp32")}


def _pair(pkg, orc, synth, name, fmt, B):
    shape = synth.SHAPES[name]
    strat, fdt = STR[fmt]
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=11, ln_random=True), fdt)
    ref = orc.OracleModel(shape, tensors, synth.param_names(shape), rescale_every=6 if fmt == "fp16" else 0,
                          weight_format=fmt, state_fp16=fmt == "fp16")
    m = pkg.Model(tensors, strat, shape=shape, max_batch=B)
    return shape, m, ref


def _close(got, want, what):
    err = float(np.abs(got - want).max())
    rel = float(np.linalg.norm(got - want) / max(np.linalg.norm(want), 1e-30))
    assert err < ABS_TOL and rel < REL_TOL, f"{what}: max-abs {err:.3e}, rel-L2 {rel:.3e}"


@pytest.mark.parametrize("name,fmt,B", [("tiny4", "fp16", 12), ("tiny4b", "int8", 20), ("tiny4", "int4", 16),
                                        ("tiny52", "fp16", 12), ("tiny50", "int8", 9), ("tiny51", "int4", 10),
                                        ("mid4", "fp16", 40), ("mid52", "int4", 150), ("mid4", "int8", 100),
                                        ("mid4", "int4", 300), ("mid52", "fp16", 70)])
def test_many_streams_match_oracle(pkg, orc, synth, name, fmt, B):
    """Stream b of a B-stream decode == the oracle fed stream b's tokens.  The stream counts walk the few-row GEMM's
    tile widths: 32 (up to 32 streams), 64, 128, 256, and two 256-stream tiles (300 streams)."""
    shape, m, ref = _pair(pkg, orc, synth, name, fmt, B)
    steps = 4
    ids = synth.token_ids(shape, steps * B, seed=9).reshape(steps, B)
    got = [m.decode(ids[t]) for t in range(steps)]
    for b in list(range(min(B, 6))) + ([B // 2 + 1] if B > 64 else []) + [B - 1]:
        ref.reset()
        for t in range(steps):
            _close(got[t][b], ref.run(int(ids[t, b])), f"{name} {fmt} stream {b} step {t}")
    m.close()


@pytest.mark.parametrize("name,fmt,B", [("tiny4b", "int4", 129), ("tiny4b", "int8", 161), ("tiny4b", "fp16", 129), ("mid4", "int8", 257),
                                        ("tiny52", "int4", 193), ("wide4", "int4", 256), ("wide4", "int8", 1030)])
def test_streams_over_pair_tiles(pkg, orc, synth, name, fmt, B):
    """More than 128 streams run on pairs of SMs: row tiles of 96 to 256 rows whose last one is ragged, 3 to 7 slices of K
    (scales taken slice by slice and four at a time, weight slots that are not full), channel tiles whose second half is
    partly or wholly outside, K cut in several pieces and, above 1024 rows, in one.  First, last and tile-edge streams."""
    shape, m, ref = _pair(pkg, orc, synth, name, fmt, B)
    ids = synth.token_ids(shape, 2 * B, seed=31).reshape(2, B)
    got = [m.decode(ids[t]) for t in range(2)]
    for b in sorted({0, 31, 95, 127, 128, B // 2, B - 1}):
        ref.reset()
        for t in range(2):
            _close(got[t][b], ref.run(int(ids[t, b])), f"{name} {fmt} stream {b} of {B} step {t}")
    m.close()


def test_int8_weight_slots_of_which_one_group_has_nothing(pkg, orc, synth):
    """int8 products whose expanders work in two groups (65 to 128 streams; more than 128 tokens, on pairs of SMs) over a range of K that
    starts at an odd slice and is long enough for the ring of weight slots to come round: its first slot holds one slice alone, the other
    group's.  Attention projections of 100 streams: three ranges of 32 slices on 148 SMs; ffn value of 200 tokens: nine of 124."""
    shape = synth.Shape("4", 1, 2048, 7936, 96)
    k1 = shape.n_embd // 64
    cuts = [z * k1 // 3 for z in range(4)]
    assert any(a % 2 == 1 and b - a >= 8 for a, b in zip(cuts, cuts[1:])), cuts
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=11, ln_random=True), "fp32")
    ref = orc.OracleModel(shape, tensors, synth.param_names(shape), rescale_every=0, weight_format="int8", state_fp16=False)
    m = pkg.Model(tensors, "cuda int8", shape=shape, max_batch=100)
    ids = synth.token_ids(shape, 2 * 100, seed=9).reshape(2, 100)
    got = [m.decode(ids[t]) for t in range(2)]
    for b in (0, 64, 99):
        ref.reset()
        for t in range(2):
            _close(got[t][b], ref.run(int(ids[t, b])), f"int8 stream {b} step {t}")
    m.reset_states()
    ref.reset()
    prompt = [int(t) for t in ids.reshape(-1)]
    _close(m.run(prompt), ref.run_seq(prompt), "int8 prompt of 200 tokens")
    m.close()


@pytest.mark.parametrize("fmt", ["fp16", "int4"])
def test_eight_streams_of_a_wide_model_take_the_gemm_path(pkg, orc, synth, fmt):
    """A model whose channel-mix width does not leave room for 8 streams in the persistent kernel's shared memory
    (8 x 8192 inputs) is still created with max_batch = 8: batches of 5..8 are decoded by the GEMM path, 1..4 by the
    persistent kernel, on the same state."""
    shape, m, ref = _pair(pkg, orc, synth, "wide4", fmt, 8)
    ids = synth.token_ids(shape, 3 * 8, seed=21).reshape(3, 8)
    got = [m.decode(ids[0]), m.decode(ids[1]), m.decode(ids[2][:3])]   # 8, 8, then 3 streams
    for b in (0, 2, 7):
        ref.reset()
        for t in range(3):
            if t == 2 and b >= 3:
                break
            _close(got[t][b], ref.run(int(ids[t, b])), f"wide4 {fmt} stream {b} step {t}")
    m.close()


@pytest.mark.parametrize("name,fmt", [("tiny4b", "fp16"), ("tiny4b", "int8"), ("tiny4b", "int4"), ("mid52", "fp16"),
                                      ("tiny50", "fp16"), ("tiny52", "int8"), ("wide4", "fp16"), ("wide4", "int4")])
def test_every_few_stream_batch_of_one_model(pkg, orc, synth, name, fmt):
    """Batches of 1 .. 5 and 8 streams of the same slots, alternating between the two persistent kernels and their
    instances, down to one stream: input widths that are not a multiple of eight 64-input chunks (some warps own none),
    and one that takes several weight tiles per row block."""
    shape, m, ref = _pair(pkg, orc, synth, name, fmt, 8)
    sizes = [8, 4, 1, 3, 2, 5, 1, 2]
    ids = synth.token_ids(shape, len(sizes) * 8, seed=5).reshape(len(sizes), 8)
    got = [m.decode(ids[t][:n]) for t, n in enumerate(sizes)]
    for b in (0, 1, 2, 4, 7):
        ref.reset()
        for t, n in enumerate(sizes):
            if b < n:
                _close(got[t][b], ref.run(int(ids[t, b])), f"{name} {fmt} stream {b} step {t} of {n} streams")
    m.close()


@pytest.mark.parametrize("C", [1024, 1088, 2112, 3136])
def test_layernorm_rows_of_every_width(pkg, orc, synth, C):
    """The LayerNorm launch shapes of few rows (256, 512 or 768 threads with one piece of the row each, 256 with several)
    at widths that leave their last warps partly idle, behind a projection that left its partial sums."""
    shape = synth.Shape("4", 2, C, 1152, 96)
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=11, ln_random=True), "fp16")
    ref = orc.OracleModel(shape, tensors, synth.param_names(shape), rescale_every=6, weight_format="fp16", state_fp16=True)
    m = pkg.Model(tensors, "cuda fp16", shape=shape, max_batch=12)
    ids = synth.token_ids(shape, 2 * 12 + 7, seed=4)
    got = [m.decode(ids[:12]), m.decode(ids[12:24])]
    prompt = m.run([int(t) for t in ids[24:]])
    for b in (11, 0):
        ref.reset()
        for t in range(2):
            _close(got[t][b], ref.run(int(ids[t * 12 + b])), f"C={C} stream {b} step {t}")
    _close(prompt, ref.run_seq([int(t) for t in ids[24:]]), f"C={C} prompt after the steps of stream 0")
    m.close()


@pytest.mark.parametrize("version,fmt,B", [("5.2", "fp16", 9), ("5.1", "int8", 17), ("5", "int4", 33), ("5.2", "int8", 130)])
def test_rwkv5_rows_add_their_slabs(pkg, orc, synth, version, fmt, B):
    """The RWKV-5 row kernel behind products whose K is cut in several pieces (1,088 inputs: 17 slices, the last piece a short
    one), with and without the gate, decay by head and by channel, up to 128 rows and above."""
    shape = synth.Shape(version, 1, 1088, 1152, 96, n_head=17)
    strat, fdt = STR[fmt]
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=11, ln_random=True), fdt)
    ref = orc.OracleModel(shape, tensors, synth.param_names(shape), rescale_every=6 if fmt == "fp16" else 0,
                          weight_format=fmt, state_fp16=fmt == "fp16")
    m = pkg.Model(tensors, strat, shape=shape, max_batch=B)
    ids = synth.token_ids(shape, 3 * B, seed=8).reshape(3, B)
    got = [m.decode(ids[t]) for t in range(3)]
    for b in (0, B // 2, B - 1):
        ref.reset()
        for t in range(3):
            _close(got[t][b], ref.run(int(ids[t, b])), f"{version} {fmt} stream {b} of {B} step {t}")
    m.close()


@pytest.mark.parametrize("vocab", [61, 1027, 16390, 40001])
def test_argmax_of_rows_with_ties(pkg, synth, vocab):
    """The arg-max of a row is found in parts: every logit turns up several times (the head repeats after 59 words), so that the
    largest one stands in several parts, and its first place is the answer.  Ragged widths, some parts with nothing to do."""
    shape = synth.Shape("4", 1, 128, 256, vocab)
    tensors = synth.generate(shape, seed=3, ln_random=True)
    tensors["head.weight"] = np.ascontiguousarray(tensors["head.weight"][:, np.arange(vocab) % 59])
    m = pkg.Model(synth.to_file_dtypes(shape, tensors, "fp16"), "cuda fp16", shape=shape, max_batch=9)
    ids = synth.token_ids(shape, 9, seed=6)
    want = m.decode(ids).argmax(1)
    m.reset_states()
    assert np.array_equal(m.decode(ids, want_logits=False, want_argmax=True), want) and want.max() < 59
    m.close()


@pytest.mark.parametrize("rows", [9, 100, 200, 300])
def test_argmax_of_rows_with_infinities_and_nan(pkg, synth, rows):
    """8, 4, 2 and 1 CTAs per row; head entries of +inf, -inf and NaN, so that rows hold infinities of either sign and NaN.  The order is
    that of the bit patterns, sign and magnitude (as in the persistent kernels): the logits of the same step say which id that is."""
    shape = synth.Shape("4", 1, 128, 256, 5001)
    tensors = synth.generate(shape, seed=3, ln_random=True)
    ids = synth.token_ids(shape, rows, seed=6)
    for cols in ({77: np.inf, 78: -np.inf}, {4990: np.nan}, {c: -np.inf for c in range(0, 5001, 2)}):
        head = tensors["head.weight"].copy()
        for c, v in cols.items():
            head[0, c] = v
        m = pkg.Model(synth.to_file_dtypes(shape, {**tensors, "head.weight": head}, "fp16"), "cuda fp16", shape=shape, max_batch=rows)
        bits = m.decode(ids).view(np.uint32)
        want = np.where(bits >> 31, ~bits, bits | 0x80000000).argmax(1)
        m.reset_states()
        assert np.array_equal(m.decode(ids, want_logits=False, want_argmax=True), want), sorted(cols)[:2]
        m.close()


@pytest.mark.parametrize("name,fmt,B", [("tiny4b", "fp16", 8), ("tiny4", "int4", 5)])
def test_a_captured_step_of_few_streams(pkg, synth, name, fmt, B):
    """5 to 8 RWKV-4 streams on a stream that is being captured: the first such step (by rows, whose buffers came with the model) can be
    captured and replayed, and agrees with the step outside a capture."""
    import ctypes
    import torch
    shape = synth.SHAPES[name]
    strat, fdt = STR[fmt]
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=11, ln_random=True), fdt)
    m = pkg.Model(tensors, strat, shape=shape, max_batch=B)
    ids = synth.token_ids(shape, B, seed=9).astype(np.int32)
    m.decode(ids[:1])           # what a first launch loads is loaded
    m.reset_states()
    got = torch.zeros(B, shape.vocab, device="cuda")
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode="thread_local")
        rc = pkg.lib().fr_b200_decode(m.handle, ids.ctypes.data_as(ctypes.c_void_p), B, ctypes.c_void_p(got.data_ptr()), None,
                                      ctypes.c_void_p(side.cuda_stream))
        graph.capture_end()
    pkg.check(rc, "captured decode")
    graph.replay()
    torch.cuda.synchronize()
    m.reset_states()
    _close(got.cpu().numpy(), m.decode(ids), f"{name} {fmt} captured")
    m.close()


def _capture(pkg, calls, keep=False):
    """The C calls of `calls(stream)`, which return their status, as one CUDA graph; nothing runs."""
    import torch
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph(keep_graph=keep)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode="thread_local")
        rcs = calls(ctypes.c_void_p(side.cuda_stream))
        graph.capture_end()
    for rc in rcs:
        pkg.check(rc, "captured call")
    return graph


@pytest.mark.parametrize("version,L,fmt,B", [("4", 1, "fp16", 1), ("4", 1, "int8", 2), ("4", 3, "fp16", 4), ("5.2", 1, "fp16", 5)])
def test_replays_of_captured_steps(pkg, synth, version, L, fmt, B):
    """Two captured steps of the persistent kernels, replayed three times with steps outside the graph in between: the bits of the
    same steps one by one.  A replay writes its exchange words with the tags of the replay before; with one layer a word is
    written once a token, so that nothing but a clear tells the two apart."""
    import torch
    shape = synth.Shape(version, L, 128, 512, 96, n_head=2 if version != "4" else 0)
    strat, fdt = STR[fmt]
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=11, ln_random=True), fdt)
    m = pkg.Model(tensors, strat, shape=shape, max_batch=B)
    ids = synth.token_ids(shape, 3 * B, seed=9).reshape(3, B).astype(np.int32)
    want = [m.decode(ids[t]) for t in (0, 1, 0, 1, 2, 2, 0, 1, 2)]
    state = [m.export_state(b) for b in range(B)]
    m.reset_states()
    got = torch.zeros(2, B, shape.vocab, device="cuda")
    graph = _capture(pkg, lambda st: [pkg.lib().fr_b200_decode(m.handle, ids[t].ctypes.data_as(ctypes.c_void_p), B,
                                                               ctypes.c_void_p(got[t].data_ptr()), None, st) for t in (0, 1)])
    have = []
    for what in ("graph", "graph", 2, 2, "graph", 2):
        if what == "graph":
            graph.replay()
            torch.cuda.synchronize()
            have.extend(got.cpu().numpy())
        else:
            have.append(m.decode(ids[what]))
    assert np.array_equal(np.stack(have), np.stack(want))
    assert all(np.array_equal(m.export_state(b), state[b]) for b in range(B))
    m.close()


@pytest.mark.parametrize("name,fmt,B", [("tiny4b", "fp16", 12), ("tiny4", "int4", 1), ("tiny52", "int8", 9), ("mid4", "int8", 200)])
def test_launch_counts(pkg, synth, name, fmt, B):
    """info()["launches"] counts the kernels of a call: the kernel nodes of the same call as a CUDA graph, for a step and for a greedy
    run (whose steps the model replays from a graph of its own outside a capture)."""
    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    shape = synth.SHAPES[name]
    strat, fdt = STR[fmt]
    m = pkg.Model(synth.to_file_dtypes(shape, synth.generate(shape, seed=11, ln_random=True), fdt), strat, shape=shape, max_batch=B)
    ids = synth.token_ids(shape, B, seed=9).astype(np.int32)
    p = ids.ctypes.data_as(ctypes.c_void_p)
    out = torch.zeros(8, B, dtype=torch.int32, device="cuda")

    def kernels(calls):
        graph = _capture(pkg, calls, keep=True)
        h, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t()
        assert cu.cuGraphGetNodes(h, None, ctypes.byref(n)) == 0
        nodes = (ctypes.c_void_p * n.value)()
        assert cu.cuGraphGetNodes(h, nodes, ctypes.byref(n)) == 0
        kinds = []
        for node in nodes:
            kind = ctypes.c_int(-1)
            assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
            kinds.append(kind.value)
        return kinds.count(0)               # CU_GRAPH_NODE_TYPE_KERNEL

    def counted(call):
        l0 = m.info()["launches"]
        call()
        return m.info()["launches"] - l0
    step = counted(lambda: m.decode(ids, want_logits=False, want_argmax=True))
    run = counted(lambda: m.decode_greedy(ids, 8))
    assert step == kernels(lambda st: [pkg.lib().fr_b200_decode(m.handle, p, B, None, ctypes.c_void_p(out.data_ptr()), st)])
    assert run == kernels(lambda st: [pkg.lib().fr_b200_decode_greedy(m.handle, p, B, 8, ctypes.c_void_p(out.data_ptr()), st)])
    m.close()


def test_captured_batches_take_the_kernel_of_the_same_step_outside(pkg, synth):
    """5 streams of RWKV-4 have the bits of the row path inside a capture, too; in a model made for more streams, whose rows are not
    there before the first step, the capture falls back to the persistent kernel, and 9 streams are refused and break no capture."""
    import torch
    shape = synth.SHAPES["tiny4b"]
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=11, ln_random=True), "fp16")
    ids = synth.token_ids(shape, 9, seed=9).astype(np.int32)
    p = ids.ctypes.data_as(ctypes.c_void_p)
    got = torch.zeros(9, shape.vocab, device="cuda")
    for max_batch in (5, 9):
        m = pkg.Model(tensors, "cuda fp16", shape=shape, max_batch=max_batch)
        refused = []

        def calls(st):
            if max_batch == 9:
                refused.append(pkg.lib().fr_b200_decode(m.handle, p, 9, ctypes.c_void_p(got.data_ptr()), None, st))
            return [pkg.lib().fr_b200_decode(m.handle, p, 5, ctypes.c_void_p(got.data_ptr()), None, st)]
        graph = _capture(pkg, calls)
        assert refused == ([-4] if max_batch == 9 else [])
        graph.replay()
        torch.cuda.synchronize()
        have = got[:5].cpu().numpy()
        m.reset_states()
        want = m.decode(ids[:5])
        assert np.array_equal(have, want) == (max_batch == 5)
        _close(have, want, f"captured, max_batch {max_batch}")
        m.close()


@pytest.mark.parametrize("name,fmt,B", [("tiny4b", "fp16", 9), ("tiny52", "int8", 9), ("tiny4", "int4", 520)])
def test_replays_of_captured_row_steps(pkg, synth, name, fmt, B):
    """Captured steps and greedy runs of the GEMM path hold their ids and their buffers: replays give the bits of the same calls one
    by one when the caller's array has other ids in it by then, and after a prompt and a greedy run have asked for larger buffers."""
    import torch
    shape = synth.SHAPES[name]
    strat, fdt = STR[fmt]
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=11, ln_random=True), fdt)
    m = pkg.Model(tensors, strat, shape=shape, max_batch=B)
    lib, n_greedy = pkg.lib(), 6
    ids = synth.token_ids(shape, 3 * B, seed=9).reshape(3, B).astype(np.int32)
    want = [m.decode(ids[t]) for t in (0, 1, 0, 1)]
    want_ids = [m.decode_greedy(ids[2], n_greedy), m.decode_greedy(ids[2], n_greedy)]
    m.reset_states()
    got = torch.zeros(2, B, shape.vocab, device="cuda")
    picked = torch.zeros(n_greedy, B, dtype=torch.int32, device="cuda")
    own = ids.copy()

    def at(t):
        return own[t].ctypes.data_as(ctypes.c_void_p)
    steps = _capture(pkg, lambda st: [lib.fr_b200_decode(m.handle, at(t), B, ctypes.c_void_p(got[t].data_ptr()), None, st) for t in (0, 1)])
    greedy = _capture(pkg, lambda st: [lib.fr_b200_decode_greedy(m.handle, at(2), B, n_greedy, ctypes.c_void_p(picked.data_ptr()), st)])
    own[:] = 1

    def replay(graph, out):
        graph.replay()
        torch.cuda.synchronize()
        return out.cpu().numpy()
    have = list(replay(steps, got))
    now = [m.export_state(b) for b in range(B)]
    m.run([int(t) for t in ids[0]] * (4000 // B))           # more rows than any call before
    m.decode_greedy(ids[0], 8)                               # and more ids
    for b in range(B):
        m.import_state(now[b], b)
    have += list(replay(steps, got))
    assert np.array_equal(np.stack(have), np.stack(want))
    assert np.array_equal(replay(greedy, picked), want_ids[0]) and np.array_equal(replay(greedy, picked), want_ids[1])
    m.close()


def test_loading_with_room_for_one_copy_of_the_weights(pkg, synth, monkeypatch):
    """Eight streams of an fp16 RWKV-4 model go by rows, from a second copy of the weights, though the persistent kernel takes them as well:
    that copy must not take the memory of a model that loads without it.  272 MiB of weights, 64 of embedding and 64 to upload the largest
    matrix: 400 MiB.  A copy of 272 made between the first two fits and leaves too little (from 544 on, below 672); made last it
    does not fit below 608, and need not."""
    import gc
    import torch
    shape = synth.Shape("4", 8, 1024, 4096, 32768)
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=11, ln_random=True), "fp16")
    ids = synth.token_ids(shape, 8, seed=9)

    def logits():
        m = pkg.Model(tensors, "cuda fp16", shape=shape, max_batch=8)
        got = m.decode(ids)
        m.close()
        return got

    want = logits()                      # what a first load leaves on the device is there
    monkeypatch.setenv("FR_B200_ROW_COPIES", "0")
    alone = logits()                     # the persistent kernel takes eight such streams
    monkeypatch.delenv("FR_B200_ROW_COPIES")
    gc.collect()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    taken = torch.empty(free - (576 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = logits()
    finally:
        del taken
        torch.cuda.empty_cache()
    assert np.array_equal(got, alone)
    _close(got, want, "persistent kernel against rows")


def test_small_and_large_batches_share_state(pkg, orc, synth):
    """The persistent kernel (<= 8 streams) and the GEMM path (> 8) read and write the same state slots, and streams
    that are decoded together need not have seen the same number of tokens (continuous batching: a stream joins a
    running batch after a reset, a prompt of its own or a few extra steps)."""
    for name in ("tiny4", "tiny52"):
        shape, m, ref = _pair(pkg, orc, synth, name, "fp16", 12)
        ids = synth.token_ids(shape, 48, seed=3).reshape(4, 12)
        fed = [[] for _ in range(12)]

        def step(row, streams):
            got = m.decode(ids[row][:streams])
            for b in range(streams):
                fed[b].append(int(ids[row, b]))
            return got
        step(0, 12)                      # 12 streams: GEMM path
        step(1, 4)                       # streams 0..3 one token further: persistent kernel
        got = step(2, 12)                # all together again, 0..3 a token ahead of 4..11
        m.reset_states(5)                # stream 5 starts over while the others are an odd number of tokens in
        fed[5] = []
        got = step(3, 12)
        for b in (0, 3, 4, 5, 11):
            ref.reset()
            for t in fed[b]:
                want = ref.run(t)
            _close(got[b], want, f"{name} stream {b} after {len(fed[b])} tokens")
        # the same through the persistent kernel: streams 0..5, stream 5 one reset behind
        m.reset_states(2)
        fed[2] = []
        got = step(0, 6)
        for b in (1, 2, 5):
            ref.reset()
            for t in fed[b]:
                want = ref.run(t)
            _close(got[b], want, f"{name} stream {b} (persistent kernel) after {len(fed[b])} tokens")
        m.close()


def test_greedy_many_streams_on_device(pkg, orc, synth):
    """decode_greedy for 16 streams == Run -> argmax -> Run on the host."""
    shape, m, ref = _pair(pkg, orc, synth, "tiny4b", "fp16", 16)
    first = [int(t) for t in synth.token_ids(shape, 16, seed=1)]
    got = m.decode_greedy(first, 5)
    m.reset_states()
    cur = np.array(first, np.int32)
    for t in range(5):
        cur = m.decode(cur).argmax(1).astype(np.int32)
        assert np.array_equal(cur, got[t])
    m.close()


@pytest.mark.parametrize("name,fmt", [("tiny4b", "fp16"), ("tiny4", "int4"), ("tiny52", "int8")])
def test_prompts_of_any_model_use_the_rows_path(pkg, orc, synth, name, fmt, monkeypatch):
    """With the W^T copies present, RWKV-4 and quantised models process prompts as GEMMs too (RWKV-4 WKV scanned per
    channel); result and state must match the oracle's token loop."""
    monkeypatch.setenv("FR_B200_SEQ_MIN", "2")
    shape, m, ref = _pair(pkg, orc, synth, name, fmt, 9)
    ids = [int(t) for t in synth.token_ids(shape, 100, seed=5)]
    launches0 = m.info()["launches"]
    got = m.run(ids)
    assert m.info()["launches"] - launches0 < 100         # not one launch per token
    _close(got, ref.run_seq(ids), f"{name} {fmt} prompt")
    _close(m.run(3), ref.run(3), f"{name} {fmt} next token")
    m.close()


def test_state_export_import_per_slot(pkg, orc, synth):
    """Every stream slot of a 12-stream model exports and imports on its own: a slot's state moved to another slot
    continues exactly as the original does, and the other slots are untouched."""
    shape, m, ref = _pair(pkg, orc, synth, "tiny52", "fp16", 12)
    ids = synth.token_ids(shape, 36, seed=13).reshape(3, 12)
    for t in range(2):
        m.decode(ids[t])
    snap = [m.export_state(b) for b in range(12)]
    m.import_state(snap[3], slot=9)                       # stream 9 becomes a copy of stream 3
    nxt = ids[2].copy()
    nxt[9] = nxt[3]
    got = m.decode(nxt)
    assert np.array_equal(got[9], got[3])
    ref.reset()
    for t in range(2):
        ref.run(int(ids[t, 3]))
    _close(got[9], ref.run(int(nxt[3])), "moved stream")
    for b in (0, 5, 11):                                  # untouched slots: export -> reset -> import restores them
        now = m.export_state(b)
        m.reset_states(b)
        m.import_state(now, slot=b)
        assert np.array_equal(m.export_state(b), now)
    m.close()
