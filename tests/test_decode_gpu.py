"""Batched TDT greedy decode on the GPU (through the C ABI) against the CPU oracle.

Bit-exactness: the token ids, frame indices and durations the GPU emits must equal what the
reference's state machine produces when it is fed the very logits the GPU computed (logit replay).
Numerics: the GPU's logits (fp32 CUDA-core path, and the three-term split-bf16 tensor-core path) must agree with
the fp32 oracle's to 1e-4 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle


def decode_gpu(ctx, encs, trace=True):
    import scriptrs_b200 as sb

    offs = np.zeros(len(encs) + 1, np.int64)
    offs[1:] = np.cumsum([e.shape[0] for e in encs])
    cat = np.concatenate([e for e in encs if e.shape[0]] or [np.zeros((0, 1024), np.float32)])
    d_enc = torch.from_numpy(np.ascontiguousarray(cat)).cuda() if cat.size else torch.zeros(1, 1024, device="cuda")
    torch.cuda.synchronize()
    tmax = int(max(e.shape[0] for e in encs))
    return sb.tdt_decode_device(ctx, d_enc.data_ptr(), offs, trace_cap=(11 * tmax + 2) if trace else 0)


@pytest.fixture(params=["tensor", "simt"], autouse=True)
def decode_path(request, ctx):
    """Every test runs on both decoders: split-bf16 tensor-core steps (default) and the fp32 persistent kernel."""
    ctx.set_option("simt_decode", 1 if request.param == "simt" else 0)
    yield request.param
    ctx.set_option("simt_decode", 0)


@pytest.fixture(scope="module")
def weights(ctx):
    import scriptrs_b200 as sb

    wn = oracle.seeded_decoder_weights(7)
    sb.load_model(ctx, wn, encoder_layers=0, has_encoder=False, has_decoder=True)
    return wn


def test_config3_replay_is_bit_exact_and_logits_match(ctx, weights):
    rng = np.random.default_rng(33)
    encs = [rng.standard_normal((126, 1024)).astype(np.float32) for _ in range(32)]
    got = decode_gpu(ctx, encs)
    w = oracle.tdt_weights_from_named(weights)
    identical = 0
    for g, enc in zip(got, encs):
        rep = oracle.greedy_replay(g["logits"], time_steps=126)
        assert rep["steps"] == g["steps"]
        assert np.array_equal(rep["tokens"], g["tokens"])
        assert np.array_equal(rep["frames"], g["frames"])
        assert np.array_equal(rep["durations"], g["durations"])
        assert np.allclose(rep["conf"], g["conf"], rtol=1e-5, atol=1e-7)
        full = oracle.tdt_decode(w, enc, want_trace=True)
        # first iteration: same inputs on both sides, so the logits must agree numerically
        a, b = g["logits"][0], full["logits"][0]
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-4
        if (len(full["tokens"]) == len(g["tokens"]) and np.array_equal(full["tokens"], g["tokens"])
                and np.array_equal(full["frames"], g["frames"]) and np.array_equal(full["durations"], g["durations"])):
            identical += 1
            n = min(len(g["logits"]), len(full["logits"]))
            assert np.abs(g["logits"][:n] - full["logits"][:n]).max() < 5e-4
    # an fp32 near-tie may flip a decision between two summation orders; it must be rare
    assert identical >= 30, identical


def test_ragged_batch_and_edge_lengths(ctx, weights):
    rng = np.random.default_rng(5)
    lens = [1, 2, 7, 0, 188, 33, 167, 1]
    encs = [rng.standard_normal((t, 1024)).astype(np.float32) for t in lens]
    got = decode_gpu(ctx, encs)
    for g, t in zip(got, lens):
        if t == 0:
            assert g["steps"] == 0 and len(g["tokens"]) == 0
            continue
        rep = oracle.greedy_replay(g["logits"], time_steps=t)
        assert rep["steps"] == g["steps"]
        for k in ("tokens", "frames", "durations"):
            assert np.array_equal(rep[k], g[k])
        assert (g["frames"] < t).all()


def test_results_do_not_depend_on_batch_composition(ctx, weights):
    rng = np.random.default_rng(9)
    a = rng.standard_normal((60, 1024)).astype(np.float32)
    b = rng.standard_normal((90, 1024)).astype(np.float32)
    alone = decode_gpu(ctx, [a], trace=False)[0]
    mixed = decode_gpu(ctx, [b, a, b, b], trace=False)
    for k in ("tokens", "frames", "durations", "conf"):
        assert np.array_equal(alone[k], mixed[1][k])
        assert np.array_equal(mixed[0][k], mixed[2][k])


def test_max_tokens_overflow_is_reported(ctx, weights):
    import scriptrs_b200 as sb

    enc = torch.randn(50, 1024, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(sb.ScriptrsError) as e:
        sb.tdt_decode_device(ctx, enc.data_ptr(), np.array([0, 50], np.int64), max_tokens=2)
    assert e.value.status == 12


def test_many_sequences_span_several_gemm_tiles(ctx, weights, decode_path):
    """300 ragged sequences: more than two 128-row tiles of the tensor-core products, and the wide-tile launch
    of the fp32 kernel; every sequence must equal its own replay and what it gives when decoded alone."""
    rng = np.random.default_rng(77)
    lens = rng.integers(1, 40, size=300)
    encs = [rng.standard_normal((int(t), 1024)).astype(np.float32) for t in lens]
    got = decode_gpu(ctx, encs)
    for g, t in zip(got, lens):
        rep = oracle.greedy_replay(g["logits"], time_steps=int(t))
        assert rep["steps"] == g["steps"]
        for k in ("tokens", "frames", "durations"):
            assert np.array_equal(rep[k], g[k])
    for i in (0, 131, 299):
        alone = decode_gpu(ctx, [encs[i]], trace=False)[0]
        for k in ("tokens", "frames", "durations", "conf"):
            assert np.array_equal(alone[k], got[i][k])


@pytest.mark.parametrize("n", [1, 8, 9, 16, 17, 33])
def test_batch_sizes_around_the_kernel_lines(ctx, weights, n):
    """One, two and more groups of eight columns, the largest batch of the few-sequences kernel and the smallest of the
    general one: a clip gives the same numbers bit for bit in each, and equals its replay."""
    rng = np.random.default_rng(n)
    lens = [int(t) for t in rng.integers(0, 30, size=n - 1)] + [41]
    encs = [rng.standard_normal((t, 1024)).astype(np.float32) for t in lens]
    fill = [rng.standard_normal((5, 1024)).astype(np.float32) for _ in range(40)]
    got = decode_gpu(ctx, encs)
    larger = decode_gpu(ctx, fill + encs, trace=False)[len(fill):]
    for g, h, t in zip(got, larger, lens):
        if t == 0:
            assert g["steps"] == h["steps"] == 0 and len(g["tokens"]) == 0
            continue
        rep = oracle.greedy_replay(g["logits"], time_steps=t)
        assert rep["steps"] == g["steps"] == h["steps"]
        for k in ("tokens", "frames", "durations", "conf"):
            assert np.array_equal(g[k], h[k])
            if k != "conf":
                assert np.array_equal(rep[k], g[k])


def test_small_cell_states_keep_their_digits(ctx, weights):
    """Candidate gates near zero (rows of the third gate scaled by 1e-4, the predictor's projection by 1e6): the hyperbolic
    tangent must be exact relative to its own size there.  Formed as a difference from one it has an absolute error of 2^-24
    or more, 1e-2 of these states and of the logits; the first step's logits are held to 2e-4 of 64-bit arithmetic: the split
    products drop 2^-16 of |x||w| in each of the chain's four, the functions and sums some 2^-21."""
    import scriptrs_b200 as sb

    w = {k: v.copy() for k, v in weights.items()}
    third = slice(2 * 640, 3 * 640)
    for k in ("weight_ih", "weight_hh", "bias_ih", "bias_hh"):
        w["predictor.lstm." + k][:, third] *= np.float32(1e-4)
    w["joint.pred.weight"] *= np.float32(1e6)
    enc = np.random.default_rng(11).standard_normal((1, 1024)).astype(np.float32)
    try:
        sb.load_model(ctx, w, encoder_layers=0, has_encoder=False, has_decoder=True)
        got = [decode_gpu(ctx, [enc] * n)[-1]["logits"][0] for n in (1, 17)]  # both kernels' cells
    finally:
        sb.load_model(ctx, weights, encoder_layers=0, has_encoder=False, has_decoder=True)
    d = {k: v.astype(np.float64) for k, v in w.items()}
    x = d["predictor.embedding"][1024]
    for layer in range(2):
        g = d["predictor.lstm.weight_ih"][layer] @ x + d["predictor.lstm.bias_ih"][layer] + d["predictor.lstm.bias_hh"][layer]
        i, _, c, o = np.split(g, 4)
        x = np.tanh(np.tanh(c) / (1.0 + np.exp(-i))) / (1.0 + np.exp(-o))
    z = d["joint.enc.weight"] @ enc[0] + d["joint.enc.bias"] + d["joint.pred.weight"] @ x + d["joint.pred.bias"]
    ref = d["joint.out.weight"] @ np.maximum(z, 0.0) + d["joint.out.bias"]
    for logits in got:
        assert np.linalg.norm(logits - ref) / np.linalg.norm(ref) < 2e-4


@pytest.mark.parametrize("blank_bias", [0.0, 1.5])
@pytest.mark.parametrize("n", [383, 384, 401, 1000])
def test_large_batches_equal_small_ones(ctx, weights, decode_path, n, blank_bias):
    """The largest batch of the kernel for some hundred sequences, and the one for more (its smallest, a last group of one column,
    more than one block of tiles per thread block): clips of 0 to 12 frames, with an emission in nearly every step or with blanks
    in most.  Tokens, confidences and logits equal those of the same clips in batches of 100, bit for bit, and their replay."""
    import scriptrs_b200 as sb

    if decode_path == "simt":
        pytest.skip("the lines are those of the tensor-core decoder")
    w = dict(weights)
    w["joint.out.bias"] = weights["joint.out.bias"].copy()
    w["joint.out.bias"][1024] += np.float32(blank_bias)
    rng = np.random.default_rng(n)
    encs = [rng.standard_normal((int(t), 1024)).astype(np.float32) for t in rng.integers(0, 13, size=n)]
    try:
        sb.load_model(ctx, w, encoder_layers=0, has_encoder=False, has_decoder=True)
        got = decode_gpu(ctx, encs)
        small = [g for i in range(0, n, 100) for g in decode_gpu(ctx, encs[i:i + 100])]
    finally:
        sb.load_model(ctx, weights, encoder_layers=0, has_encoder=False, has_decoder=True)
    for i, (g, h) in enumerate(zip(got, small)):
        assert g["steps"] == h["steps"]
        for k in ("tokens", "frames", "durations", "conf"):
            assert np.array_equal(g[k], h[k]), (i, k)
        assert np.array_equal(g["logits"], h["logits"]), i
        if i % 17 == 0 and encs[i].shape[0]:
            rep = oracle.greedy_replay(g["logits"], time_steps=encs[i].shape[0])
            assert rep["steps"] == g["steps"] and all(np.array_equal(rep[k], g[k]) for k in ("tokens", "frames", "durations"))


def test_two_contexts_decode_at_the_same_time(ctx, weights, decode_path):
    """The decoder's grid occupies every SM and waits for itself.  Two host threads with a context each keep it busy with batches
    of all three kernels: every call must return what it returns alone."""
    import threading

    import scriptrs_b200 as sb

    rng = np.random.default_rng(5)
    batches = [[rng.standard_normal((int(t), 1024)).astype(np.float32) for t in rng.integers(1, 30, size=n)] for n in (400, 5, 60)]
    second = sb.Context(0)
    try:
        second.set_option("simt_decode", 1 if decode_path == "simt" else 0)
        sb.load_model(second, weights, encoder_layers=0, has_encoder=False, has_decoder=True)
        alone = [decode_gpu(ctx, b, trace=False) for b in batches]
        results, errors = {}, []

        def work(who, c):
            try:
                for i in range(12):
                    results[who, i] = decode_gpu(c, batches[(i + who) % 3], trace=False)
            except Exception as e:  # noqa: BLE001
                errors.append(e)

        threads = [threading.Thread(target=work, args=(k, c)) for k, c in enumerate((ctx, second))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors
        for (who, i), got in results.items():
            for g, a in zip(got, alone[(i + who) % 3]):
                assert all(np.array_equal(g[k], a[k]) for k in ("tokens", "frames", "durations", "conf"))
    finally:
        second.close()
