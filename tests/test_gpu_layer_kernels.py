"""One token routed inside the FFN kernel, passes of the GEMM kernels wider than an accumulator buffer, router logits of large
batches, hidden rows of any size: sizes and values at which each changes its way, against the CPU oracle."""
import numpy as np
import pytest

import mer_b200
import oracle

pytestmark = pytest.mark.gpu
synth = __import__("importlib").import_module("mer_b200.synth")

FFN_TOL = 1e-3  # max-abs error relative to the RMS of the reference output


def rel_rms_err(got, ref):
    ref = np.asarray(ref, np.float64)
    return float(np.max(np.abs(np.asarray(got, np.float64) - ref)) / (np.sqrt(np.mean(ref ** 2)) + 1e-30))


def backend(dtype, D, F, n_experts, **kw):
    stride = (256 + mer_b200.expert_bytes(dtype, D, F) + 4095) // 4096 * 4096
    return mer_b200.Backend(dtype, D, F, stride * n_experts, n_experts, **kw)


def ffn_reference(dtype, blobs, x, F, ids, w):
    """The routed sum for a given routing."""
    return sum(np.float32(wi) * oracle.expert_forward(dtype, blobs[i], x, x.size, F) for i, wi in zip(ids, w))


# one down item a CTA (short rows of few experts) and several; 128 and 129, 256 and 257 experts; 32 slots; odd widths
@pytest.mark.parametrize("dtype", [oracle.Q8_0, oracle.Q4_0])
@pytest.mark.parametrize("E,k,D,F,groups,shared", [
    (128, 8, 2048, 768, 1, False), (129, 8, 256, 96, 1, False), (256, 8, 1024, 256, 8, True), (257, 4, 64, 32, 1, False),
    (40, 32, 256, 64, 1, False), (33, 31, 96, 160, 1, True), (4, 1, 4128, 288, 1, False), (3, 2, 512, 4096, 1, True), (1, 1, 32, 32, 1, False)])
def test_one_token_layers(dtype, E, k, D, F, groups, shared):
    rng = np.random.default_rng(E + D)
    blobs = [synth.make_expert_blob(dtype, D, F, 101, 0, e) for e in range(min(E, 12))]
    blobs = [blobs[e % len(blobs)] for e in range(E + shared)]
    W = rng.standard_normal((E, D)).astype(np.float32) * 0.1
    sigmoid = groups > 1
    bias = (rng.standard_normal(E) * 0.1).astype(np.float32) if sigmoid else None
    og = oracle.LinearGate(W, E, D, k, scoring_func=int(sigmoid), correction_bias=bias, n_group=groups, topk_group=max(1, groups // 2))
    with backend(dtype, D, F, 2 * E + 1 + shared, max_tokens=4, max_top_k=k + shared) as b:
        for layer in range(2):  # ids of the second layer do not start at zero
            for e in range(E):
                b.admit(layer * E + e, 1, blobs[e], wait=e == E - 1)
            mer_b200.LinearGate.with_routing(W, E, D, k, int(sigmoid), True, bias, groups, max(1, groups // 2), 1.0).bind(b, layer, *([2 * E] if shared else []))
        if shared:
            b.admit(2 * E, 1, blobs[E])
        for i in range(6):  # plain launches, then replayed ones
            x = rng.standard_normal((1, D)).astype(np.float32)
            out, ids, w = b.moe_layer_forward(i % 2, x)
            rids, rw = og.route(x[0])[:2]
            assert set(ids[0].tolist()) == set(rids.tolist())
            order = np.argsort(ids[0]), np.argsort(rids)
            # an error d of a logit is one of d, relatively, of its weight; fp32 sums of D terms are good to about 1e-6 of the logits' size
            assert np.allclose(w[0][order[0]], rw[order[1]], rtol=8e-6 * (1 + 0.1 * np.sqrt(D)))
            ref = ffn_reference(dtype, blobs, x[0], F, ids[0], w[0])
            if shared:
                ref = ref + oracle.expert_forward(dtype, blobs[E], x[0], D, F)
            assert rel_rms_err(out[0], ref) <= FFN_TOL


def test_one_token_with_a_missing_expert_fails_closed_and_the_next_call_works():
    dtype, E, k, D, F = oracle.Q8_0, 128, 8, 256, 64
    W = synth.make_router(E, D, 103)
    blob = synth.make_expert_blob(dtype, D, F, 103, 0, 0)
    with backend(dtype, D, F, E, max_tokens=4, max_top_k=k) as b:
        for e in range(1, E):
            b.admit(e, 1, blob)
        gate = mer_b200.LinearGate(W, E, D, k)
        gate.bind(b, 0)
        og = oracle.LinearGate(W, E, D, k)
        x = synth.make_activations(400, D, 103)
        hits = [t for t in range(400) if 0 in og.route(x[t])[0]]
        free = [t for t in range(400) if t not in hits]
        for t in (hits[0], free[0], hits[1], free[1]):
            if t in hits:
                with pytest.raises(mer_b200.GpuExpertDispatchError) as e:
                    b.moe_layer_forward(0, x[t:t + 1])
                assert e.value.kind == mer_b200.GpuExpertDispatchErrorKind.ResidencyMiss
            else:
                out, ids, w = b.moe_layer_forward(0, x[t:t + 1])
                assert rel_rms_err(out[0], ffn_reference(dtype, [blob] * E, x[t], F, ids[0], w[0])) <= FFN_TOL


# Tokens of very small and very large values: gate, up and hidden values scale with them (SiLU is linear in its limits).  Values of one row that lie far apart, and rows
# far below their bounds, are in test_gpu_hidden_values.py.
@pytest.mark.parametrize("n_tokens", [1, 4, 9])
@pytest.mark.parametrize("scale", [1e-18, 1.0, 1e15])
def test_hidden_rows_of_any_magnitude(n_tokens, scale):
    dtype, D, F = oracle.Q8_0, 256, 2048
    blob = synth.make_expert_blob(dtype, D, F, 104, 0, 0)
    x = synth.make_activations(n_tokens, D, 104) * np.float32(scale)
    with backend(dtype, D, F, 2, max_tokens=16) as b:
        b.admit(1, 1, blob)
        b.set_kernel_path(2)
        got = b.expert_forward_f32(0, 1, x)
    for t in range(n_tokens):
        ref = oracle.expert_forward(dtype, blob, x[t], D, F, oracle.FWD_AUTHORITATIVE)
        assert rel_rms_err(got[t], ref) <= FFN_TOL


# The rule takes passes of up to 256 tokens from 37 experts of these shapes on: groups of one wide pass, of a wide and a narrow one, of
# unequal ones, beside groups of a few tokens.
@pytest.mark.parametrize("dtype", [oracle.Q4_0, oracle.Q8_0])
def test_passes_of_two_accumulator_buffers(dtype):
    E, D, F = 38, 4096, 2048
    sizes = [129, 256, 257, 400, 144, 16, 1, 130] + [1] * 30
    rng = np.random.default_rng(105)
    blobs = [synth.make_expert_blob(dtype, D, F, 105, 0, e) for e in range(3)]
    which = np.concatenate([np.full(n, e) for e, n in enumerate(sizes)])
    rng.shuffle(which)
    T = which.size
    W = np.zeros((E, D), np.float32)
    W[np.arange(E), np.arange(E)] = 10.0
    x = rng.standard_normal((T, D)).astype(np.float32) * 0.5
    x[:, :E] = 0.0
    x[np.arange(T), which] = 3.0
    with backend(dtype, D, F, E, max_tokens=T, max_top_k=1) as b:
        for e in range(E):
            b.admit(e, 1, blobs[e % 3], wait=e == E - 1)
        mer_b200.LinearGate(W, E, D, 1).bind(b, 0)
        out, ids, _ = b.moe_layer_forward(0, x)
        again, _, _ = b.moe_layer_forward(0, x)
        b.set_kernel_path(2)
        other, _, _ = b.moe_layer_forward(0, x)
    assert (ids[:, 0] == which).all() and np.array_equal(out, again)
    for e, n in enumerate(sizes[:8]):
        for t in np.flatnonzero(which == e)[[0, n // 2, n - 1]]:
            ref = oracle.expert_forward(dtype, blobs[e % 3], x[t], D, F)
            assert rel_rms_err(out[t], ref) <= FFN_TOL
    rms = np.sqrt((other.astype(np.float64) ** 2).mean(1, keepdims=True))
    assert np.max(np.abs(out - other) / rms) <= FFN_TOL  # the two kernel families, every row


# partial expert tiles (8 a fragment tile, 64 and 128 a CTA), partial token tiles of 128, slices of K, one chunk of a slice; both sides of the rule that takes
# fp32 tiles, those of 32 x 64 and of 64 x 128; tokens that are selected four a CTA
@pytest.mark.parametrize("E,k,T,D", [(17, 2, 256, 256), (60, 6, 257, 512), (64, 8, 383, 2304), (65, 4, 300, 1024), (128, 8, 385, 2048), (129, 8, 256, 7168),
                                     (256, 8, 511, 1280), (128, 8, 320, 2048), (128, 8, 321, 2048), (128, 4, 1600, 256), (2050, 8, 256, 256), (2050, 4, 300, 512)])
def test_router_logits_of_large_batches(E, k, T, D):
    F, dtype = 32, oracle.Q8_0
    rng = np.random.default_rng(E)
    W = (rng.standard_normal((E, D)) * 0.05).astype(np.float32)
    x = (rng.standard_normal((T, D)) * np.exp(rng.uniform(-4, 1, (T, 1)))).astype(np.float32)  # rows of very different size
    blob = np.zeros(mer_b200.expert_bytes(dtype, D, F), np.uint8)
    with backend(dtype, D, F, E, max_tokens=T, max_top_k=k) as b:
        for e in range(E):
            b.admit(e, 1, blob, wait=e == E - 1)
        mer_b200.LinearGate(W, E, D, k).bind(b, 0)
        _, ids, w = b.moe_layer_forward(0, x)
    s = x.astype(np.float64) @ W.astype(np.float64).T
    top = -np.sort(-s, axis=1)
    # fp32 sums of D terms are good to about 1e-6 of the terms' root sum of squares, and softmax scores to a few units of 2^-24: closer
    # logits have two right orders
    noise = 1e-6 * np.sqrt((x.astype(np.float64) ** 2).sum(1)) * 0.05 + 5e-7
    picked = np.take_along_axis(s, ids.astype(np.int64), 1)
    assert (picked >= top[:, k - 1:k] - noise[:, None]).all() and all(len(set(r)) == k for r in ids.tolist())
    p = np.exp(picked - picked.max(1, keepdims=True))
    ref = p / p.sum(1, keepdims=True)
    # an error d of a logit is one of d, relatively, of its weight
    assert (np.abs(w - ref) <= ref * (4 * noise[:, None] + 1e-6)).all()


# Values far above the rest of their router row (at columns where the tokens are zero) or of their token (where the router is): the logits come from the
# small ones alone, and are as good as without the large ones.
@pytest.mark.parametrize("where,power", [("router", 10), ("router", 15), ("router", 20), ("router", 26), ("router", 40), ("token", 10), ("token", 20), ("token", 26)])
def test_router_logits_beside_values_far_above_the_others(where, power):
    E, k, T, D, F, dtype = 64, 8, 700, 2048, 32, oracle.Q8_0  # (the parts: what a thread of the fp32 tiles would add is long enough)
    rng = np.random.default_rng(power)
    W = (rng.standard_normal((E, D)) * 0.05).astype(np.float32)
    x = rng.standard_normal((T, D)).astype(np.float32)
    far = rng.permutation(D)[:16]  # one of 64 neighbours, or a few
    W[:, far], x[:, far] = 0.0, 0.0
    if where == "router":
        W[:, far] = 0.05 * 2.0 ** power * rng.choice([-1.0, 1.0], (E, 16))
    else:
        x[:, far] = 2.0 ** power
    blob = np.zeros(mer_b200.expert_bytes(dtype, D, F), np.uint8)
    with backend(dtype, D, F, E, max_tokens=T, max_top_k=k) as b:
        for e in range(E):
            b.admit(e, 1, blob, wait=e == E - 1)
        mer_b200.LinearGate(W, E, D, k).bind(b, 0)
        ids, w = b.route(0, x)
    s = x.astype(np.float64) @ W.astype(np.float64).T
    # fp32 sums of D terms are good to about 1e-6 of the terms' root sum of squares, softmax scores to a few units of 2^-24
    noise = 1e-6 * np.sqrt(D) * 0.05 + 5e-7
    picked = np.take_along_axis(s, ids.astype(np.int64), 1)
    assert (picked >= -np.sort(-s, axis=1)[:, k - 1:k] - noise).all() and all(len(set(r)) == k for r in ids.tolist())
    p = np.exp(picked - picked.max(1, keepdims=True))
    ref = p / p.sum(1, keepdims=True)
    assert (np.abs(w - ref) <= ref * (4 * noise + 1e-6)).all()


def test_router_logits_of_tokens_that_are_not_finite():
    # sigmoid scores of infinite logits are 0 and 1: the batch must select what the same tokens select alone
    E, k, T, D, F, dtype = 32, 4, 300, 256, 32, oracle.Q8_0
    rng = np.random.default_rng(9)
    W = rng.standard_normal((E, D)).astype(np.float32)
    x = rng.standard_normal((T, D)).astype(np.float32) * 0.01
    x[7, 3], x[8, 5], x[131, 0], x[299, 255] = np.inf, -np.inf, np.inf, np.nan
    x[9] = 0.0
    x[10] *= 1e30
    blob = np.zeros(mer_b200.expert_bytes(dtype, D, F), np.uint8)
    with backend(dtype, D, F, E, max_tokens=T, max_top_k=k) as b:
        for e in range(E):
            b.admit(e, 1, blob, wait=e == E - 1)
        gate = mer_b200.LinearGate.with_routing(W, E, D, k, 1, True, None, 1, 1, 1.0)
        gate.bind(b, 0)
        ids, w = b.route(0, x)
        for t in (7, 8, 9, 10, 11, 131, 299):
            one, w1 = b.route(0, x[t:t + 1])
            assert np.array_equal(np.sort(ids[t]), np.sort(one[0])), t
            assert np.allclose(np.sort(w[t]), np.sort(w1[0]), rtol=1e-5, equal_nan=True), t
