"""Sizes at which the dispatch changes its way of routing, grouping, multiplying or moving host data, against the CPU oracle."""
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


@pytest.mark.parametrize("E,k,B,D,F", [
    (8, 2, 16, 64, 32), (8, 2, 17, 64, 32),        # 32 pairs are grouped in one warp, more in a block
    (4, 1, 2048, 64, 32), (4, 1, 2049, 64, 32),    # the block's largest number of pairs
    (512, 1, 40, 64, 32), (513, 1, 40, 64, 32),    # and of groups
    (512, 32, 4, 64, 32), (64, 16, 3, 64, 32),     # the same with passes of four
    (3, 1, 1, 1024, 32), (100, 2, 5, 1024, 32),    # one and two expert rows per router CTA
    (16, 1, 300, 1024, 32), (17, 1, 300, 1024, 32),  # logits of a large batch: direct, in small tiles,
    (128, 1, 1921, 512, 32),                       # in large ones
    (2, 1, 4100, 128, 128), (130, 2, 4100, 64, 32),  # and grouped over the grid
])
def test_routing_and_grouping_edges(E, k, B, D, F):
    dtype = oracle.Q8_0 if B % 2 else oracle.Q4_0
    blobs = [synth.make_expert_blob(dtype, D, F, 91, 0, e) for e in range(E)]
    W = synth.make_router(E, D, 91)
    x = synth.make_activations(B, D, 91)
    with backend(dtype, D, F, E, max_tokens=B, max_top_k=k) as b:
        for e in range(E):
            b.admit(e, 1, blobs[e])
        mer_b200.LinearGate(W, E, D, k).bind(b, 0)
        out, ids, _ = b.moe_layer_forward(0, x)
    ref, rids, _, _ = oracle.moe_layer_forward(dtype, oracle.LinearGate(W, E, D, k), blobs, x, F, n_threads=8)
    same = (ids == rids).all(axis=1)  # scores within rounding of each other may swap
    assert np.count_nonzero(~same) <= B // 1000
    assert rel_rms_err(out[same], ref[same]) <= FFN_TOL


@pytest.mark.parametrize("dtype", [oracle.Q8_0, oracle.Q4_0])
@pytest.mark.parametrize("D,F,n_tokens", [(128, 128, 1), (384, 128, 65), (128, 128, 128), (384, 256, 129), (128, 384, 257)])
def test_gemm_pass_widths_and_odd_tile_counts(dtype, D, F, n_tokens):
    blob = synth.make_expert_blob(dtype, D, F, 92, 0, 0)
    x = synth.make_activations(n_tokens, D, 92)
    with backend(dtype, D, F, 2, max_tokens=max(n_tokens, 16)) as b:
        b.admit(1, 1, blob)
        b.set_kernel_path(3)
        got = b.expert_forward_f32(0, 1, x)
    ref = np.stack([oracle.expert_forward(dtype, blob, x[t], D, F, oracle.FWD_AUTHORITATIVE) for t in range(n_tokens)])
    assert rel_rms_err(got, ref) <= FFN_TOL


@pytest.mark.parametrize("n_tokens", [897, 1025])  # passes of unequal width
def test_a_row_gives_the_same_bits_in_every_pass_of_a_large_group(n_tokens):
    dtype, D, F = oracle.Q8_0, 256, 128
    blob = synth.make_expert_blob(dtype, D, F, 96, 0, 0)
    rows = synth.make_activations(7, D, 96)
    which = np.arange(n_tokens) % 7
    with backend(dtype, D, F, 1, max_tokens=n_tokens) as b:
        b.admit(0, 1, blob)
        b.set_kernel_path(3)
        got = b.expert_forward_f32(0, 0, rows[which])
    ref = np.stack([oracle.expert_forward(dtype, blob, r, D, F, oracle.FWD_AUTHORITATIVE) for r in rows])
    assert rel_rms_err(got[:7], ref) <= FFN_TOL
    assert np.array_equal(got, got[:7][which])


# pairs grouped in one block by atomics (streaming and GEMM kernels), and over the grid
@pytest.mark.parametrize("E,k,B,path", [(16, 4, 40, 2), (16, 4, 200, 3), (4, 2, 4100, 2), (4, 2, 4100, 3)])
def test_a_grouping_whose_order_the_atomics_decide_gives_the_same_bits_every_time(E, k, B, path):
    dtype, D, F = oracle.Q4_0, 256, 128
    W = synth.make_router(E, D, 97)
    x = synth.make_activations(B, D, 97)
    x[1::2] = x[0:-1:2][:x[1::2].shape[0]]  # pairs of equal rows lie side by side
    with backend(dtype, D, F, E, max_tokens=B, max_top_k=k) as b:
        for e in range(E):
            b.admit(e, 1, synth.make_expert_blob(dtype, D, F, 97, 0, e))
        mer_b200.LinearGate(W, E, D, k).bind(b, 0)
        b.set_kernel_path(path)
        first, ids, w = b.moe_layer_forward(0, x)
        for _ in range(5):
            again, ids2, w2 = b.moe_layer_forward(0, x)
            assert np.array_equal(first, again) and np.array_equal(ids, ids2) and np.array_equal(w, w2)
    n = B // 2 * 2
    assert np.array_equal(first[0:n:2], first[1:n:2])


@pytest.mark.parametrize("dtype", [oracle.Q8_0, oracle.Q4_0])
@pytest.mark.parametrize("D,F,n_tokens", [(32, 96, 3), (96, 544, 9), (160, 32, 8), (4128, 288, 5), (7168, 256, 12)])
def test_streaming_remainders_of_four_blocks_and_of_sixteen_tiles(dtype, D, F, n_tokens):
    blob = synth.make_expert_blob(dtype, D, F, 93, 0, 0)
    x = synth.make_activations(n_tokens, D, 93) + 0.5  # block sums far from zero: the zero point's share matters
    with backend(dtype, D, F, 2, max_tokens=n_tokens) as b:
        b.admit(1, 1, blob)
        b.set_kernel_path(2)
        got = b.expert_forward_f32(0, 1, x)
    ref = np.stack([oracle.expert_forward(dtype, blob, x[t], D, F, oracle.FWD_AUTHORITATIVE) for t in range(n_tokens)])
    assert rel_rms_err(got, ref) <= FFN_TOL


@pytest.mark.parametrize("B", [1, 64, 65])  # 64 rows of 256 values are moved by kernels, 65 by copies
def test_repeated_host_calls_read_new_rows(B):
    dtype, E, D, F, k = oracle.Q8_0, 16, 256, 64, 4
    blobs = [synth.make_expert_blob(dtype, D, F, 94, 0, e) for e in range(E)]
    W = synth.make_router(E, D, 94)
    gate = oracle.LinearGate(W, E, D, k)
    with backend(dtype, D, F, E, max_tokens=B, max_top_k=k) as b:
        for e in range(E):
            b.admit(e, 1, blobs[e])
        mer_b200.LinearGate(W, E, D, k).bind(b, 0)
        for rep in range(5):  # plain launches, then the capture, then replays
            x = synth.make_activations(B, D, 95 + rep)
            ref, rids, rw, _ = oracle.moe_layer_forward(dtype, gate, blobs, x, F, n_threads=8)
            ids, w = b.route(0, x)
            assert (ids == rids).all() and np.allclose(w, rw, rtol=1e-5, atol=1e-7)
            out, ids, _ = b.moe_layer_forward(0, x)
            assert (ids == rids).all() and rel_rms_err(out, ref) <= FFN_TOL
            assert rel_rms_err(b.moe_step_weighted_into(0, x[0], rids[0], rw[0]), ref[0]) <= FFN_TOL


@pytest.mark.parametrize("D,F,E,k,B,path", [(96, 160, 4, 2, 3, 0), (1024, 32, 8, 2, 5, 0), (256, 128, 4, 2, 300, 0), (45, 37, 4, 2, 3, 0),
                                            (256, 256, 4, 2, 40, 3), (64, 96, 4, 2, 7, 1)])
@pytest.mark.parametrize("block", [False, True])
def test_device_rows_may_start_on_any_float(D, F, E, k, B, path, block):
    import torch
    dtype = oracle.Q8_0
    x = synth.make_activations(B, D, 98)
    with backend(dtype, D, F, E, max_tokens=B, max_top_k=k) as b:
        for e in range(E):
            b.admit(e, 1, synth.make_expert_blob(dtype, D, F, 98, 0, e))
        mer_b200.LinearGate(synth.make_router(E, D, 98), E, D, k).bind(b, 0)
        if block:
            b.install_layer(0, np.linspace(0.5, 1.5, D, dtype=np.float32), 1e-6, residual=True)
        b.set_kernel_path(path)
        results = []
        for shift in (0, 1, 2, 3):
            d_x = torch.zeros(B * D + 4, device="cuda")[shift:shift + B * D]
            d_out = torch.zeros(B * D + 4, device="cuda")
            d_x.copy_(torch.from_numpy(x.reshape(-1)))
            for rep in range(4):  # plain launches, the capture, a replay
                d_out.fill_(7.0)
                b.moe_layer_forward_device(0, d_x.data_ptr(), B, d_out.data_ptr() + 4 * shift, torch.cuda.current_stream().cuda_stream)
                b.stream_check(0, torch.cuda.current_stream().cuda_stream)
                got = d_out.cpu().numpy()
                assert (got[:shift] == 7.0).all() and (got[shift + B * D:] == 7.0).all()
                results.append(got[shift:shift + B * D])
        assert np.isfinite(results[0]).all() and all(np.array_equal(results[0], r) for r in results)


@pytest.mark.parametrize("dtype,D,F", [(oracle.Q8_0, 96, 32), (oracle.Q4_0, 256, 256), (oracle.Q4_0, 45, 37)])
def test_a_device_payload_may_start_on_any_byte(dtype, D, F):
    import torch
    blob = synth.make_expert_blob(dtype, D, F, 99, 0, 0)
    x = synth.make_activations(2, D, 99)
    with backend(dtype, D, F, 4, max_tokens=2) as b:
        for shift in range(4):
            buf = torch.zeros(blob.size + 4, dtype=torch.uint8, device="cuda")
            buf[shift:shift + blob.size].copy_(torch.from_numpy(blob))
            torch.cuda.synchronize()
            b.admit_device(shift, 1, buf.data_ptr() + shift, blob.size)
        got = [b.expert_forward_f32(0, e, x) for e in range(4)]
    ref = np.stack([oracle.expert_forward(dtype, blob, r, D, F) for r in x])
    assert rel_rms_err(got[0], ref) <= FFN_TOL and all(np.array_equal(got[0], g) for g in got)


@pytest.mark.parametrize("D,E,n", [(32, 16, 1), (96, 24, 5), (736, 16, 7), (1056, 40, 3), (1280, 130, 9), (5376, 160, 17)])
def test_router_logits_of_widths_that_are_no_multiple_of_1024(D, E, n):
    # a warp's slice of a row is D / 32 groups of four values: fewer than its lanes, a ragged last step, many steps
    k = 4
    rng = np.random.default_rng([7, D, E])
    W, x = (rng.standard_normal((E, D)) * 0.02).astype(np.float32), rng.standard_normal((n, D)).astype(np.float32)
    stride = (256 + mer_b200.expert_bytes(mer_b200.DTYPE_Q8_0, D, 32) + 4095) // 4096 * 4096
    with mer_b200.Backend(mer_b200.DTYPE_Q8_0, D, 32, stride, E, max_tokens=n, max_top_k=k) as b:
        mer_b200.LinearGate(W, E, D, k).bind(b, 0)
        ids, w = b.route(0, x)
    logits = x.astype(np.float64) @ W.astype(np.float64).T
    p = np.exp(logits - logits.max(1, keepdims=True))
    # a lane adds D / 256 products (four at a time), the warp five sums, the CTA eight: so many roundings of at most the terms' magnitude
    err = ((D / 256 + 14) * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ np.abs(W).T.astype(np.float64))).max(1)
    for t in range(n):
        best = np.argsort(-logits[t], kind="stable")
        if np.diff(-logits[t][best[:k + 1]]).min() <= 2 * err[t]:
            continue  # a tie within rounding has two right answers
        assert ids[t].tolist() == best[:k].tolist()
        want = p[t][best[:k]] / p[t][best[:k]].sum()
        assert (np.abs(w[t] - want) <= want * (4 * err[t] + 2e-6)).all()


@pytest.mark.parametrize("D,E,n", [
    (1056, 128, 40), (736, 160, 24), (2848, 24, 300),                    # four expert rows a CTA, slices that end short of a warp, or of several
    (1056, 128, 80), (736, 160, 100), (5376, 160, 100), (2848, 24, 400),  # eight
    (1280, 8, 2048), (1280, 8, 2049), (1280, 12, 1030), (2816, 16, 1024), (2816, 16, 1025), (2816, 3, 256),  # few experts: 512 CTAs, and the GEMM behind
    (7168, 32, 600), (4096, 32, 300), (4096, 33, 300),  # partial sums of up to 32 experts, a value a lane, and of more
    (256, 437, 256), (256, 512, 256), (256, 683, 256), (64, 1000, 9), (64, 1366, 8),  # shared memory with the kernels' tables on either side of 48 KB
])
def test_router_logits_of_several_rows_a_cta(D, E, n):
    k = min(4, E // 2) if E > 3 else 2
    rng = np.random.default_rng([8, D, E, n])
    W, x = (rng.standard_normal((E, D)) * 0.02).astype(np.float32), rng.standard_normal((n, D)).astype(np.float32)
    bad = [1, 6, n // 2, n - 1]  # a NaN, infinities: their own rows only
    x_bad = x.copy()
    x_bad[bad[0], D - 1], x_bad[bad[1], 0], x_bad[bad[2], D // 2], x_bad[bad[3], 33] = np.nan, np.inf, -np.inf, np.nan
    stride = (256 + mer_b200.expert_bytes(mer_b200.DTYPE_Q8_0, D, 32) + 4095) // 4096 * 4096
    with mer_b200.Backend(mer_b200.DTYPE_Q8_0, D, 32, stride, 2 * E, max_tokens=n, max_top_k=k) as b:
        mer_b200.LinearGate(W, E, D, k).bind(b, 0)
        ids, w = b.route(0, x)
        mer_b200.LinearGate.with_routing(W, E, D, k, 1, True, None, 1, 1, 1.0).bind(b, 1)  # sigmoid: the softmax of a NaN is an error
        clean, mixed = b.route(1, x), b.route(1, x_bad)
        alone = [b.route(1, x_bad[t:t + 1]) for t in bad]
    good = np.setdiff1d(np.arange(n), bad)
    assert (clean[0][good] == mixed[0][good]).all() and (clean[1][good] == mixed[1][good]).all()
    for t, (i1, w1) in zip(bad, alone):
        assert np.array_equal(np.sort(mixed[0][t]), np.sort(i1[0])) and np.allclose(np.sort(mixed[1][t]), np.sort(w1[0]), rtol=1e-5, equal_nan=True)
    logits = x.astype(np.float64) @ W.astype(np.float64).T
    p = np.exp(logits - logits.max(1, keepdims=True))
    # the roundings of the test above; the logits GEMM adds 32 terms a thread, or operands of 22 bits by eights, eight slices or warps and up to 16 parts of K
    roundings = D / 256 + (14 if D % 256 or n < 256 or (E <= 16 and -(-E // 8) * -(-n // 4) <= 512) else 64)
    err = (roundings * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ np.abs(W).T.astype(np.float64))).max(1)
    best = np.argsort(-logits, axis=1, kind="stable")
    clear = np.diff(-np.take_along_axis(logits, best[:, :k + 1], 1), axis=1).min(1) > 2 * err
    assert clear.mean() > 0.8  # of the others, ties within rounding, either answer is right
    assert (ids[clear] == best[clear, :k]).all()
    want = np.take_along_axis(p, best[:, :k], 1)
    want /= want.sum(1, keepdims=True)
    assert (np.abs(w - want) <= want * (4 * err[:, None] + 2e-6))[clear].all()
