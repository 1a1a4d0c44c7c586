"""bonsai_b200_linear in one launch and in two: the same y and the same Q8_1 scratch, bit for bit, where CTAs, clusters, row segments and
the rule's ranges end; and the calls that only two launches answer.  (Two launches against the oracle: test_linear_one_call and the mat-vec's tests.)"""
import pytest

from captured import launches

pytestmark = pytest.mark.gpu


def operands(gpu, n_out, n_in, signed, seed=3):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    W = torch.empty(n_out * (n_in // 128) * 34, dtype=torch.uint8, device="cuda")
    assert gpu.synth_pq2_0(W, 0, n_out * (n_in // 128), seed) == 0
    signs = torch.randint(0, 2, (n_in,), generator=g, device="cuda").float() * 2 - 1 if signed else None
    return W, torch.randn(n_in, generator=g, device="cuda"), signs


def outputs(gpu, W, x, signs, n_out, n_in, fuse, y=None):
    """(y, scratch) of a call with the option at `fuse`, and how many kernels it is."""
    import torch
    y = torch.full((n_out + 2,), float("nan"), device="cuda")[1:-1] if y is None else y
    xq = torch.zeros(n_in // 32 * 36, dtype=torch.uint8, device="cuda")
    try:
        assert gpu.set_option("fuse_linear", fuse) == 0
        kernels = launches(lambda: gpu.linear(W, x, signs, y, xq, n_out, n_in))
    finally:
        gpu.set_option("fuse_linear", -1)
    return y, xq, len(kernels)


# rows: less than a quad, a quad and one, all CTAs of one launch and one more; the last row of the one-launch form and the first behind it
@pytest.mark.parametrize("n_in,n_out,kernels", [
    (1024, 1, 1), (1024, 592, 1), (1024, 593, 1), (1024, 5920, 1), (1024, 5921, 1), (1024, 9001, 1), (2048, 5, 1), (2048, 5920, 1), (2048, 5921, 2), (3072, 529, 1), (3072, 3168, 1),
    (3072, 3169, 2), (4096, 37, 1), (4096, 1920, 1), (4096, 1921, 2), (5120, 7, 1), (5120, 480, 1), (5120, 481, 1), (5120, 1024, 1), (5120, 1920, 1), (5120, 1921, 2), (6144, 1001, 1), (6144, 1080, 1),
    (6144, 1081, 2), (7168, 840, 1), (7168, 841, 2), (8192, 479, 1), (8192, 960, 1), (8192, 961, 2), (9216, 64, 2), (17408, 33, 2)])
@pytest.mark.parametrize("signed", [False, True])
def test_same_bits_as_two_launches(gpu, n_in, n_out, kernels, signed):
    import torch
    W, x, signs = operands(gpu, n_out, n_in, signed)
    y2, xq2, n2 = outputs(gpu, W, x, signs, n_out, n_in, 0)
    y1, xq1, n1 = outputs(gpu, W, x, signs, n_out, n_in, -1)
    assert n2 == 2 and n1 == kernels
    assert torch.equal(y1, y2) and torch.equal(xq1, xq2)
    assert gpu.device_status() == 0


@pytest.mark.parametrize("n", [1024, 2048])
@pytest.mark.parametrize("over", ["x", "signs", "scratch"])
def test_output_over_its_input(gpu, n, over):
    """y over x or the signs: the whole vector is read first, as by two launches.  The scratch over the signs of 1024 values, likewise."""
    import torch
    if over == "scratch" and n > 1024:
        pytest.skip("several CTAs of the quantiser read and write it")
    W, x, signs = operands(gpu, n, n, True)
    want, xq, _ = outputs(gpu, W, x, signs, n, n, 0)
    y, scratch = torch.empty(n, device="cuda"), torch.empty_like(xq)
    if over == "x":
        y = x
    elif over == "signs":
        y = signs
    else:
        scratch = signs.view(torch.uint8)
    assert gpu.linear(W, x, signs, y, scratch, n, n) == 0
    assert torch.equal(y, want) and torch.equal(scratch[:xq.numel()], xq)


def test_unaligned_vector(gpu):
    import torch
    W, x, signs = operands(gpu, 100, 5120, True)
    want, xq, _ = outputs(gpu, W, x, signs, 100, 5120, -1)
    odd = torch.empty(5121, device="cuda")
    odd[1:].copy_(x)
    got, xq_odd, kernels = outputs(gpu, W, odd[1:], signs, 100, 5120, -1)
    assert kernels == 2 and torch.equal(got, want) and torch.equal(xq, xq_odd)


def test_refused_clusters(gpu):
    """Where a launch in clusters is refused two launches serve, from then on without trying; one block of 1024 needs no cluster."""
    import torch
    W, x, signs = operands(gpu, 100, 5120, True)
    want, _, kernels = outputs(gpu, W, x, signs, 100, 5120, -1)
    assert kernels == 1
    try:
        assert gpu.set_option("refuse_clusters", 1) == 0
        for _ in range(2):
            got, _, kernels = outputs(gpu, W, x, signs, 100, 5120, -1)
            assert kernels == 2 and torch.equal(got, want)
        assert outputs(gpu, W, x[:1024].clone(), None, 100, 1024, -1)[2] == 1
    finally:
        gpu.set_option("refuse_clusters", 0)
    assert outputs(gpu, W, x, signs, 100, 5120, -1)[2] == 1
