"""The one-launch kernel behind mer_expert_forward_noalloc, at the sizes where it can go wrong: rows that start off a 16-byte
boundary, one block, several K ranges with a short last one, more and fewer tiles than CTAs, one to eight tokens."""
import importlib

import numpy as np
import pytest

import mer_b200
import oracle

pytestmark = pytest.mark.gpu
synth = importlib.import_module("mer_b200.synth")


@pytest.mark.parametrize("dtype,D,F,n", [
    (mer_b200.DTYPE_Q4_0, 32, 32, 1), (mer_b200.DTYPE_Q4_0, 96, 160, 4), (mer_b200.DTYPE_Q4_0, 256, 512, 5),
    (mer_b200.DTYPE_Q4_0, 4352, 288, 8), (mer_b200.DTYPE_Q4_0, 256, 4864, 3), (mer_b200.DTYPE_Q8_0, 64, 96, 8),
    (mer_b200.DTYPE_Q8_0, 2304, 288, 2), (mer_b200.DTYPE_Q8_0, 512, 2336, 7), (mer_b200.DTYPE_Q8_0, 2048, 768, 4)])
def test_flat_expert_matches_the_oracle(dtype, D, F, n):
    import torch
    blob = synth.make_expert_blob(dtype, D, F, 91, 0, 0)
    x = synth.make_activations(n, D, 91)
    x[0] *= 1e-3
    d_blob, d_x = torch.from_numpy(blob).cuda(), torch.from_numpy(x).cuda()
    d_out = torch.full((n, D), float("nan"), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(2):
        mer_b200.expert_forward_noalloc(dtype, D, F, d_blob.data_ptr(), d_x.data_ptr(), n, d_out.data_ptr(), 0.0, stream)
    torch.cuda.synchronize()
    got = d_out.cpu().numpy()
    for t in range(n):
        ref = oracle.expert_forward(dtype, blob, x[t], D, F)
        assert np.abs(got[t] - ref).max() <= 1e-3 * np.sqrt(np.mean(ref.astype(np.float64) ** 2))


@pytest.mark.parametrize("dtype,D,F,n", [
    (mer_b200.DTYPE_Q4_0, 4800, 4896, 4), (mer_b200.DTYPE_Q4_0, 2560, 7168, 1), (mer_b200.DTYPE_Q8_0, 3200, 2080, 2), (mer_b200.DTYPE_Q8_0, 4864, 2560, 4)])
def test_steps_of_two_tiles_over_several_ranges(dtype, D, F, n):
    # up to four tokens a warp multiplies two tiles at a time: CTAs with one, two, three and more of them in either phase, ranges whose last one has
    # a single block (K of 65 blocks) or a few, rows on and off a 16-byte boundary
    test_flat_expert_matches_the_oracle(dtype, D, F, n)


@pytest.mark.parametrize("dtype,D,F,n", [(mer_b200.DTYPE_Q4_0, 2048, 4096, 3), (mer_b200.DTYPE_Q8_0, 4096, 1408, 8)])
def test_a_wait_that_runs_out_is_reported_once_and_leaves_nan(dtype, D, F, n):
    # a limit of one nanosecond: the CTAs that arrive first give up on the others
    import torch
    blob = synth.make_expert_blob(dtype, D, F, 92, 0, 0)
    x = synth.make_activations(n, D, 92)
    d_blob, d_x = torch.from_numpy(blob).cuda(), torch.from_numpy(x).cuda()
    d_out = torch.zeros((n, D), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    args = (dtype, D, F, d_blob.data_ptr(), d_x.data_ptr(), n, d_out.data_ptr(), 0.0)
    mer_b200.expert_noalloc_check(stream)  # nothing is pending
    mer_b200.expert_forward_noalloc_bounded(*args, 1, stream)
    with pytest.raises(mer_b200.GpuExpertDispatchError) as e:
        mer_b200.expert_noalloc_check(stream)
    assert e.value.kind == mer_b200.GpuExpertDispatchErrorKind.Timeout
    assert np.isnan(d_out.cpu().numpy()).any(axis=1).all()  # in every row
    mer_b200.expert_noalloc_check(stream)  # reported once
    mer_b200.expert_forward_noalloc(*args, stream)  # and the next call is whole
    mer_b200.expert_noalloc_check(stream)
    ref = np.stack([oracle.expert_forward(dtype, blob, r, D, F) for r in x])
    assert np.abs(d_out.cpu().numpy() - ref).max() <= 1e-3 * np.sqrt(np.mean(ref.astype(np.float64) ** 2))


@pytest.mark.parametrize("n", [1, 4, 5, 8])
@pytest.mark.parametrize("dtype,D,F", [(mer_b200.DTYPE_Q4_0, 4128, 1056), (mer_b200.DTYPE_Q4_0, 1056, 4128), (mer_b200.DTYPE_Q8_0, 2080, 2336), (mer_b200.DTYPE_Q8_0, 512, 2304),
                                       (mer_b200.DTYPE_Q4_0, 256, 256), (mer_b200.DTYPE_Q4_0, 2048, 2048), (mer_b200.DTYPE_Q4_0, 2048, 2304), (mer_b200.DTYPE_Q4_0, 2304, 512)])
def test_ranges_that_leave_warps_without_a_block(dtype, D, F, n):
    # a last range of one block (129 of Q4_0, 65 of Q8_0), of a few, and first ones of 33 or 16: the other warps make no fragments and add zeros,
    # whatever the range before left them; Q4_0 rows off a 16-byte boundary take one tile at a time, those of up to 2048 values ranges of 64 blocks
    test_flat_expert_matches_the_oracle(dtype, D, F, n)
