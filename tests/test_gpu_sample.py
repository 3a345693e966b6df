"""Device-side sampling against a numpy restatement of Sampler::Sample (sampler.cpp:38-101) + the CPU softmax it
calls (kernels/cpu/softmax.cpp:6-21), oracle/sampler_ref.py, itself pinned against the reference's own sampler compiled
from its sources: same logits, same uniform draw -> same token."""
import numpy as np
import pytest

from oracle.sampler_ref import minstd_uniforms as _minstd_uniforms, pick_distance, ref_sample

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("temperature,top_k,top_p", [(1.0, 0, 0.9), (0.7, 20, 0.95), (2.0, 5, 1.0), (1.0, 1, 0.5),
                                                     (0.05, 0, 0.3), (1.3, 0, 1.0)])
def test_sample_matches_reference_sampler(pkg, synth, temperature, top_k, top_p):
    shape = synth.SHAPES["tiny4b"]
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=4, ln_random=True), "fp16")
    B = 12
    m = pkg.Model(tensors, "cuda fp16", shape=shape, max_batch=B)
    rng = np.random.default_rng(17)
    checked = 0
    for step in range(3):
        logits = m.decode(synth.token_ids(shape, B, seed=step))
        u = rng.uniform(0, 1, B).astype(np.float32)
        got = m.sample(B, temperature, top_k, top_p, u)
        for b in range(B):
            want, margin = ref_sample(logits[b], temperature, top_k, top_p, u[b])
            if margin > 1e-5:
                assert got[b] == want, (step, b, int(got[b]), want, margin)
                checked += 1
    assert checked >= 3      # draws too close to a threshold to survive a different summation order are skipped
    # greedy corner: top_k = 1 is the arg-max whatever the draw (sampler.cpp:71-74)
    logits = m.decode(synth.token_ids(shape, B, seed=9))
    assert np.array_equal(m.sample(B, 1.0, 1, 1.0, rng.uniform(0, 1, B).astype(np.float32)), logits.argmax(1))
    m.close()


def test_sample_single_stream_after_run(pkg, synth):
    """After Model.run on stream 0 (persistent kernel) the logits are where fr_b200_sample looks for them."""
    shape = synth.SHAPES["tiny4"]
    tensors = synth.to_file_dtypes(shape, synth.generate(shape, seed=4, ln_random=True), "fp16")
    m = pkg.Model(tensors, "cuda fp16", shape=shape)
    logits = m.run(5)
    want, margin = ref_sample(logits, 1.0, 0, 0.8, 0.37)
    got = m.sample(1, 1.0, 0, 0.8, [0.37])
    assert margin < 1e-5 or got[0] == want
    m.close()


@pytest.mark.parametrize("temperature,top_k,top_p", [(1.0, 0, 0.9), (0.7, 20, 0.95), (2.0, 0, 1.0), (1.0, 1, 0.3)])
def test_sample_matches_the_reference_sampler_binary_at_full_vocab(pkg, synth, tmp_path, temperature, top_k, top_p):
    """The reference's own Sampler::Sample + CPU softmax (sampler.cpp, kernels/cpu/softmax.cpp compiled from where they
    lie into the driver binary, `--sample` mode) against fr_b200_sample on the same logits at vocab 65536, seeded
    std::minstd_rand0 draws, with frequency / presence penalties applied on the device (fr_b200_logits_add) and on the
    host copy alike (chat.cpp:57-61)."""
    import os
    import subprocess
    exe = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle", "_ref", "fr_ref_run")
    if not os.path.exists(exe):
        pytest.skip("reference sampler not built (needs the reference tree at build time)")
    shape = synth.Shape("4", 1, 64, 64, 65536)
    master = synth.generate(shape, seed=3, ln_random=True)
    master["head.weight"] = master["head.weight"] * 6.0          # peaked logits, as a trained model's
    tensors = synth.to_file_dtypes(shape, master, "fp16")
    B, draws, seed = 4, 8, 42
    m = pkg.Model(tensors, "cuda fp16", shape=shape, max_batch=B)
    logits = m.decode(synth.token_ids(shape, B, seed=1)).copy()
    # penalties: a few tokens per stream, logit -= frequency * occurrence + presence
    rng = np.random.default_rng(5)
    streams = np.repeat(np.arange(B), 3).astype(np.int32)
    tokens = np.concatenate([np.argsort(-logits[b])[:3] for b in range(B)]).astype(np.int32)
    deltas = -(0.2 * rng.integers(1, 4, len(tokens)) + 0.2).astype(np.float32)
    m.logits_add(streams, tokens, deltas)
    for s, t, d in zip(streams, tokens, deltas):
        logits[s, t] += d
    lf = str(tmp_path / "logits.bin")
    logits.astype(np.float32).tofile(lf)
    r = subprocess.run([exe, "--sample", lf, str(shape.vocab), str(B), str(temperature), str(top_k), str(top_p), str(seed), str(draws)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    theirs = np.array([[int(x) for x in line.split()[2:]] for line in r.stdout.splitlines() if line.startswith("sample")])
    assert theirs.shape == (B, draws)
    us = _minstd_uniforms(seed, draws)
    checked = 0
    for d in range(draws):
        got = m.sample(B, temperature, top_k, top_p, [us[d]] * B)
        for b in range(B):
            want, margin = ref_sample(logits[b], temperature, top_k, top_p, np.float32(us[d]))
            assert want == theirs[b, d] or margin <= 1e-5       # the numpy restatement agrees with the reference binary
            # the device sums up to 65536 weights in segments, the reference serially: a draw closer than 1e-4 (relative
            # to the total) to a threshold may resolve to a neighbouring entry -- never further away than that
            if margin > 1e-4:
                assert got[b] == theirs[b, d], (d, b, int(got[b]), int(theirs[b, d]), margin)
                checked += 1
            else:
                dist = pick_distance(logits[b], temperature, top_k, top_p, np.float32(us[d]), int(got[b]))
                assert dist <= 1e-4, (d, b, int(got[b]), int(theirs[b, d]), margin, dist)
    # a flat distribution over the whole vocabulary (temperature 2, no cuts) gives every token ~1e-5 of the weight: all of
    # its draws are "near a threshold" and are covered by the distance check alone
    flat = top_k == 0 and top_p >= 1.0 and temperature > 1.0
    assert flat or checked >= B * draws // 2
    m.close()


@pytest.mark.parametrize("vocab", [65536, 50277])
@pytest.mark.parametrize("gain", [0.0, 0.002, 1.0, 8.0])
def test_sample_finds_its_entry_at_any_spread_of_the_logits(pkg, synth, vocab, gain):
    """All logits equal (the entry is found by its index), packed within a few thousandths (several narrowings), spread
    like untrained and like trained logits; with and without the two cuts.  Every pick lies within rounding of where the
    reference's walk over the sorted probabilities stops."""
    shape = synth.Shape("4", 1, 64, 64, vocab)
    master = synth.generate(shape, seed=3, ln_random=True)
    master["head.weight"] = master["head.weight"] * np.float32(gain)
    B = 5
    m = pkg.Model(synth.to_file_dtypes(shape, master, "fp32"), "cuda int8", shape=shape, max_batch=B)
    logits = m.decode(synth.token_ids(shape, B, seed=1)).copy()
    tol = 1e-4 if gain > 0.5 else 5e-4        # of the fp32 running sum of tens of thousands of equal probabilities
    rng = np.random.default_rng(5)
    for temperature, top_k, top_p in ((1.0, 0, 0.9), (0.7, 3000, 0.95), (2.0, 0, 0.99), (1.0, 0, 1.0), (0.3, 40, 0.999), (5.0, 1, 1.0)):
        u = rng.uniform(0, 1, B).astype(np.float32)
        u[0] = 0.0
        got = m.sample(B, temperature, top_k, top_p, u)
        assert np.array_equal(got, m.sample(B, temperature, top_k, top_p, u))
        for b in range(B):
            want, margin = ref_sample(logits[b], temperature, top_k, top_p, u[b])
            if margin > tol:
                assert got[b] == want, (temperature, top_k, top_p, b, int(got[b]), want, margin)
            else:
                assert pick_distance(logits[b], temperature, top_k, top_p, u[b], int(got[b])) <= tol
    m.close()


def _given_logits(pkg, synth, rows):
    """A model whose device logits are exactly `rows` [B, V]: a zero head, then the values as adjustments (0 + x)."""
    B, V = rows.shape
    shape = synth.Shape("4", 1, 64, 64, V)
    master = synth.generate(shape, seed=3, ln_random=True)
    master["head.weight"] = master["head.weight"] * np.float32(0)
    m = pkg.Model(synth.to_file_dtypes(shape, master, "fp16"), "cuda fp16", shape=shape, max_batch=B)
    m.decode(np.zeros(B, np.int32), want_logits=False, want_argmax=True)
    m.logits_add(np.repeat(np.arange(B), V), np.tile(np.arange(V), B), rows.reshape(-1))
    return m


@pytest.mark.parametrize("masked", [0, 1, 40000])
@pytest.mark.parametrize("top_k,top_p", [(3000, 1.5), (3000, 0.0), (0, 0.5), (0, 1.5), (60000, 2.0)])
def test_sample_with_masked_logits(pkg, synth, masked, top_k, top_p):
    """Logits of -inf are never picked and take no part in a cut, and top_p > 1 is no cut at all (the running sum does not
    reach it, sampler.cpp:59-66).  The rows have a peak far above a bulk that only a temperature above 1 gives weight to, so
    that the top-k cut falls far behind the last entry with a noticeable probability."""
    V, B = 65536, 3
    rng = np.random.default_rng(8)
    rows = (-33 - 20 * rng.random((B, V))).astype(np.float32)
    for b in range(B):
        rows[b, rng.permutation(V)[:masked]] = -np.inf
        rows[b, 17 + b] = 0.0
    m = _given_logits(pkg, synth, rows)
    for temperature in (5.0, 1.0):
        for u in ([0.0, 0.5, 0.9], [0.97, 0.7, 1.0]):
            u = np.float32(u)
            got = m.sample(B, temperature, top_k, top_p, u)
            for b in range(B):
                assert np.isfinite(rows[b, got[b]])
                # the fp32 running sum over tens of thousands of entries: 1e-3 of the total bounds its error
                dist = pick_distance(rows[b], temperature, top_k, top_p, u[b], int(got[b]))
                assert dist <= 1e-3, (temperature, top_k, top_p, b, float(u[b]), int(got[b]), dist)
    m.close()


def test_sample_of_rows_without_an_ordinary_maximum(pkg, synth):
    """+inf entries are the maximum, a row of -inf alone is a row of equals, NaN is never picked next to a number."""
    V = 4096
    rows = np.zeros((4, V), np.float32)
    rows[0, [5, 99]] = np.inf
    rows[1] = -np.inf
    rows[2, ::2] = np.nan
    rows[3] = np.nan
    m = _given_logits(pkg, synth, rows)
    for top_k, top_p in ((0, 1.0), (10, 0.9), (3, 2.0)):
        for u in (0.0, 0.4, 1.0):
            got = m.sample(4, 1.0, top_k, top_p, [u] * 4)
            assert got[0] in (5, 99)
            assert 0 <= got[1] < V and (top_k == 0 or got[1] < top_k)
            assert got[2] % 2 == 1
            assert got[3] == 0
    m.close()


@pytest.mark.parametrize("rows", [1, 512, 513, 700])
def test_sample_from_and_to_host_and_device_memory(pkg, synth, rows):
    """Draws as kernel parameters (up to 512 rows on the host) and through device memory (more rows, or given there), ids to
    the host and to the device: the same picks, and the reference's."""
    import ctypes
    import torch
    shape = synth.Shape("4", 1, 64, 64, 1000)
    master = synth.generate(shape, seed=3, ln_random=True)
    master["head.weight"] = master["head.weight"] * np.float32(4)
    m = pkg.Model(synth.to_file_dtypes(shape, master, "fp16"), "cuda fp16", shape=shape, max_batch=rows)
    logits = m.decode(np.arange(rows) % shape.vocab)
    u = np.random.default_rng(2).random(rows).astype(np.float32)
    want = m.sample(rows, 1.0, 0, 0.8, u)
    checked = 0
    for b in range(rows):
        ref, margin = ref_sample(logits[b], 1.0, 0, 0.8, u[b])
        if margin > 1e-5:
            assert want[b] == ref
            checked += 1
    assert checked >= rows * 3 // 4
    ud, out = torch.from_numpy(u).cuda(), np.empty(rows, np.int32)
    od = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    f = ctypes.c_float
    for up in (u.ctypes.data, ud.data_ptr()):
        for op in (out.ctypes.data, od.data_ptr()):
            out[:] = -1
            od.fill_(-1)
            torch.cuda.synchronize()
            pkg.check(pkg.lib().fr_b200_sample(m.handle, rows, f(1.0), 0, f(0.8), up, op, None), "fr_b200_sample")
            torch.cuda.synchronize()
            got = out if op == out.ctypes.data else od.cpu().numpy()
            assert np.array_equal(got, want)
    m.close()
