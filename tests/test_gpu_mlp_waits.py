"""The tensor-core kernels' error path: a wait that expires is reported, the
committed products are waited for, and the network stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one row tile and more tiles than SMs of the resident form; rings of one slab
# past K = 256, of their own length and longer
@pytest.mark.parametrize("M,N,K", [(128, 32, 64), (128 * 310, 256, 256), (128, 96, 320), (256, 256, 512), (1280, 256, 4096)])
def test_an_expired_wait_is_reported_and_drained(M, N, K):
    import threepoint_gb300 as tp
    import torch

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randint(-8, 9, (M, K), generator=g, device="cuda").to(torch.bfloat16)
    B = torch.randint(-8, 9, (N, K), generator=g, device="cuda").to(torch.bfloat16)
    C = torch.full((M, N), float("nan"), device="cuda")
    torch.cuda.synchronize()
    net = tp.MLP(max_batch=128)
    try:
        for _ in range(3):
            assert tp.lib().tp_mlp_set_wait_limit(net._h, 0) == tp.TP_OK
            with pytest.raises(tp.ThreepointError) as e:
                net.gemm_device(A, B, C)
            assert e.value.status == tp.TP_ERR_CUDA and "limit" in str(e.value)
            torch.cuda.synchronize()
            assert bool(torch.isnan(C).all())  # no epilogue
        assert tp.lib().tp_mlp_set_wait_limit(net._h, -1) == tp.TP_OK
        net.gemm_device(A, B, C)
        # products of integers up to 64, sums below 2^24: exact
        assert bool((C.double() == A.double() @ B.double().T).all())
    finally:
        net.close()


def test_an_expired_wait_of_a_training_step():
    import threepoint_gb300 as tp
    import torch

    rng = np.random.default_rng(1)
    net = tp.MLP(max_batch=1024)
    try:
        net.set_params(rng.standard_normal(net.param_count()) * 0.05)
        x = torch.tensor(rng.uniform(-1, 1, (1000, 8)), dtype=torch.float32, device="cuda")
        t = torch.tensor(rng.standard_normal(1000), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        assert tp.lib().tp_mlp_set_wait_limit(net._h, 0) == tp.TP_OK
        net.train_step_device(x, t, 0.0)
        with pytest.raises(tp.ThreepointError):
            net.sync()
        assert tp.lib().tp_mlp_set_wait_limit(net._h, -1) == tp.TP_OK
        net.train_step_device(x, t, 0.0)
        net.sync()
    finally:
        net.close()


def test_misaligned_operands_are_refused():
    """before a launch that would copy them in 16-byte pieces"""
    import threepoint_gb300 as tp
    import torch

    a = torch.zeros(128 * 64 + 8, dtype=torch.bfloat16, device="cuda")
    b = torch.zeros(32 * 64 + 8, dtype=torch.bfloat16, device="cuda")
    c = torch.zeros((128, 32), device="cuda")
    net = tp.MLP(max_batch=128)
    try:
        for i, j in ((1, 0), (0, 4), (3, 2)):
            with pytest.raises(tp.ThreepointError) as e:
                net.gemm_device(a[i:i + 128 * 64].view(128, 64), b[j:j + 32 * 64].view(32, 64), c)
            assert e.value.status == tp.TP_ERR_ARG
        net.gemm_device(a[8:].view(128, 64), b[8:].view(32, 64), c)
    finally:
        net.close()
