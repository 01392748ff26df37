"""Hidden values of the streaming kernels: experts whose gates saturate below zero, where SiLU leaves values many orders of magnitude below
max |gate| * max |up|, with K of either projection split and not, against the CPU oracle."""
import importlib

import numpy as np
import pytest

import mer_b200
import oracle

pytestmark = pytest.mark.gpu
synth = importlib.import_module("mer_b200.synth")

FFN_TOL = 1e-3  # max-abs error relative to the RMS of the reference output


def rel_rms_err(got, ref):
    ref = np.asarray(ref, np.float64)
    return float(np.max(np.abs(np.asarray(got, np.float64) - ref)) / np.sqrt(np.mean(ref ** 2)))


def saturated_blob(dtype, D, F, gate, seed, rows=None):
    """An expert whose gates are within a tenth of `gate` (< 0) for positive rows of mean 1, in all hidden rows or in the first `rows`."""
    blob = synth.make_expert_blob(dtype, D, F, seed, 0, 0)
    rows = F if rows is None else rows
    bb = synth.BLOCK_BYTES[dtype]
    g = blob[:F * D // 32 * bb].reshape(F, D // 32, bb)[:rows]
    # The lowest quant, as a quantiser gives a block's largest weight.  Kernels add (q + zero point) * x and -zero point * x in fp32, good to 2^-24 of the sum
    # of either's magnitudes; with quants of -1 that is 128 (Q8_0) times the gate, 5e-4 at -60, and as much relatively of SiLU.
    scale = np.random.default_rng(seed).uniform(0.9, 1.1, (rows, 1)) * (-gate / D / (8 if dtype == oracle.Q4_0 else 127))
    g[:, :, :2] = np.broadcast_to(scale.astype(np.float16), (rows, D // 32))[..., None].view(np.uint8)
    g[:, :, 2:] = 0x00 if dtype == oracle.Q4_0 else 0x81  # -8, -127
    return blob


def positive_rows(n, D, seed):
    return np.random.default_rng(seed).uniform(0.5, 1.5, (n, D)).astype(np.float32)


def backend(dtype, D, F, n_experts, **kw):
    stride = (256 + mer_b200.expert_bytes(dtype, D, F) + 4095) // 4096 * 4096
    return mer_b200.Backend(dtype, D, F, stride * n_experts, n_experts, **kw)


# K of gate/up whole (8, 9 blocks) and split (64, 128); of down whole (3, 8) and split, with a short last part (44); passes of four tokens and of
# eight; one down item a CTA (one token) and several
@pytest.mark.parametrize("dtype", [oracle.Q8_0, oracle.Q4_0])
@pytest.mark.parametrize("D,F", [(256, 2048), (288, 96), (2048, 768), (4096, 256), (2048, 1408), (512, 14336)])
@pytest.mark.parametrize("n_tokens", [1, 4, 9])
def test_saturated_gates(dtype, D, F, n_tokens):
    x = positive_rows(n_tokens, D, 11)
    gates = [-8.0, -16.0, -24.0, -60.0]
    blobs = [saturated_blob(dtype, D, F, g, 20 + i) for i, g in enumerate(gates)] + [saturated_blob(dtype, D, F, -24.0, 30, F // 2)]
    with backend(dtype, D, F, len(blobs), max_tokens=16) as b:
        b.set_kernel_path(2)
        for e, blob in enumerate(blobs):
            b.admit(e, 1, blob)
            got = b.expert_forward_f32(0, e, x)
            for t in range(n_tokens):
                assert rel_rms_err(got[t], oracle.expert_forward(dtype, blob, x[t], D, F)) <= FFN_TOL, (e, t)


# the same through a layer: one token whose experts the FFN kernel selects itself (short rows) or the router kernel does, and a small batch
@pytest.mark.parametrize("dtype", [oracle.Q8_0, oracle.Q4_0])
@pytest.mark.parametrize("D,F", [(2048, 768), (512, 4096)])
@pytest.mark.parametrize("n_tokens", [1, 6])
def test_layers_whose_experts_all_saturate(dtype, D, F, n_tokens):
    E, k = 16, 2
    blobs = [saturated_blob(dtype, D, F, -20.0, 40 + i) for i in range(3)]
    W = synth.make_router(E, D, 41)
    og = oracle.LinearGate(W, E, D, k)
    x = positive_rows(n_tokens, D, 42)
    with backend(dtype, D, F, E, max_tokens=8, max_top_k=k) as b:
        for e in range(E):
            b.admit(e, 1, blobs[e % 3])
        mer_b200.LinearGate(W, E, D, k).bind(b, 0)
        b.set_kernel_path(2)
        out, ids, w = b.moe_layer_forward(0, x)
    for t in range(n_tokens):
        assert set(ids[t].tolist()) == set(og.route(x[t])[0].tolist())
        ref = sum(np.float64(wi) * oracle.expert_forward(dtype, blobs[i % 3], x[t], D, F) for i, wi in zip(ids[t], w[t]))
        assert rel_rms_err(out[t], ref) <= FFN_TOL


# non-finite hidden values reach every output of their token and no other
@pytest.mark.parametrize("dtype", [oracle.Q8_0, oracle.Q4_0])
@pytest.mark.parametrize("n_tokens", [1, 5])
def test_hidden_values_that_are_not_finite(dtype, n_tokens):
    D, F = 512, 4096
    blob = synth.make_expert_blob(dtype, D, F, 50, 0, 0)
    x = synth.make_activations(n_tokens, D, 50)
    x[0] *= np.float32(1e25)  # gate * up is beyond fp32
    with backend(dtype, D, F, 1, max_tokens=16) as b:
        b.set_kernel_path(2)
        b.admit(0, 1, blob)
        got = b.expert_forward_f32(0, 0, x)
    assert not np.isfinite(got[0]).any()
    for t in range(1, n_tokens):
        assert rel_rms_err(got[t], oracle.expert_forward(dtype, blob, x[t], D, F)) <= FFN_TOL


# Where the device refuses cooperative launches every step is a kernel of its own: the same values, added in the same order.
@pytest.mark.parametrize("dtype", [oracle.Q8_0, oracle.Q4_0])
@pytest.mark.parametrize("D,F,E,k,n_tokens,shared", [
    (2048, 768, 24, 8, 1, False), (4096, 288, 9, 2, 1, True), (512, 14336, 4, 2, 3, False), (256, 2048, 40, 4, 9, True), (288, 96, 12, 3, 70, False)])
def test_steps_in_kernels_of_their_own(dtype, D, F, E, k, n_tokens, shared):
    blobs = [synth.make_expert_blob(dtype, D, F, 60, 0, e) for e in range(3)]
    W = synth.make_router(E, D, 61)
    x = synth.make_activations(n_tokens, D, 61)
    with backend(dtype, D, F, E + 1, max_tokens=n_tokens, max_top_k=k + 1) as b:
        for e in range(E + 1):
            b.admit(e, 1, blobs[e % 3], wait=e == E)
        mer_b200.LinearGate(W, E, D, k).bind(b, 0, *([E] if shared else []))
        results = []
        for path in (2, 4):
            b.set_kernel_path(path)
            results += [b.moe_layer_forward(0, x) for _ in range(4)]  # plain launches, then replayed ones
            one = b.moe_step_weighted_into(0, x[0], results[0][1][0], results[0][2][0])
            results[-1] += (one,)
    for out, ids, w, *_ in results:
        assert np.array_equal(out, results[0][0]) and np.array_equal(ids, results[0][1]) and np.array_equal(w, results[0][2])
    assert np.array_equal(results[3][3], results[7][3])
    for t in {0, n_tokens // 2, n_tokens - 1}:
        ref = sum(np.float64(wi) * oracle.expert_forward(dtype, blobs[i % 3], x[t], D, F) for i, wi in zip(results[0][1][t], results[0][2][t]))
        if shared:
            ref = ref + oracle.expert_forward(dtype, blobs[E % 3], x[t], D, F)
        assert rel_rms_err(results[4][0][t], ref) <= FFN_TOL
