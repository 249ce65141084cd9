"""The two-launch training step of the Lorenz-96 proposal (csrc/train.cu) where
its tiles can go wrong: one row, a partial tile, a whole one, one row more, two
tiles, and a data set whose arrays are not 16-byte aligned.  The gradient is
held to the CPU oracle's restatement with the tolerance the other gradient test
states (BF16 operands, FP32 sums)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, seed, offset=0):
    """(x_t, x_{t+1}, y_{t+1}) rows on the GPU; offset: floats into the allocation."""
    import torch

    rng = np.random.default_rng(seed)
    x = (2.3 + 3.6 * rng.standard_normal((n, 40))).astype(np.float32)
    out = []
    for v in (x, x + 0.1 * rng.standard_normal(x.shape).astype(np.float32),
              x + rng.standard_normal(x.shape).astype(np.float32)):
        buf = torch.zeros(n * 40 + offset, dtype=torch.float32, device="cuda")
        buf[offset:] = torch.as_tensor(v.reshape(-1)).cuda()
        out.append(buf[offset:].view(n, 40))
    return out


@pytest.mark.parametrize("B", [1, 127, 128, 129, 256, 148 * 128 + 1])
def test_gradient_matches_oracle_at_tile_edges(cuda, B):
    import torch
    from libbi_b200 import LearnedProposal, ModelL96
    from libbi_b200 import _native as N
    from oracle.mlp_oracle import bf16, loss_grad

    p = LearnedProposal(ModelL96(dim=40), 0.05, max(B, 128), 3)
    rng = np.random.default_rng(B)
    P = (p.params()[0] + 0.05 * rng.standard_normal(p.params()[0].size)).astype(np.float32)
    p.set_params(P)
    U = bf16(rng.standard_normal((B, 80)).astype(np.float32))
    r0 = (0.1 * rng.standard_normal((B, 40))).astype(np.float32)
    Ud, r0d = torch.as_tensor(U).to(torch.bfloat16).cuda(), torch.as_tensor(r0).cuda()
    g = torch.zeros(P.size, dtype=torch.float32, device="cuda")
    loss = ctypes.c_double()
    N.check(N.lib().bpf_proposal_loss_grad(p.handle, Ud.data_ptr(), r0d.data_ptr(), B, ctypes.byref(loss),
                                           g.data_ptr()), "bpf_proposal_loss_grad")
    want_loss, want = loss_grad(P, U, r0)
    np.testing.assert_allclose(loss.value, want_loss, rtol=1e-4)
    got, o = g.cpu().numpy().astype(np.float64), 0
    for n in (128 * 80, 128, 128 * 128, 128, 80 * 128, 80):
        a, b = got[o:o + n], want[o:o + n]
        assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b) + 1e-9
        o += n
    p.close()


@pytest.mark.parametrize("offset", [0, 1])
def test_unaligned_data_trains_alike(cuda, offset):
    """The same rows from 16-byte aligned arrays and from arrays one float on:
    the same losses and parameters bit for bit."""
    from libbi_b200 import LearnedProposal, ModelL96

    out = []
    for off in (0, offset):
        p = LearnedProposal(ModelL96(dim=40), 0.05, 512, 5)
        x, x1, y = _data(1000, 7, off)
        p.set_data(x, x1, y)
        P0 = p.params()[0]
        out.append((p.train(3, 300, 1e-3), p.params()[0]))
        p.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    assert np.isfinite(out[0][0]).all() and (out[0][1] != P0).any()


def test_workspace_follows_the_capacity(cuda):
    """Eight proposals for batches of 128 rows, one share of the gradient each
    (147 KB): far less device memory than the 148 shares of a full GPU (22 MB
    each)."""
    import torch
    from libbi_b200 import LearnedProposal, ModelL96

    LearnedProposal(ModelL96(dim=40), 0.05, 128, 1).close()
    free0 = torch.cuda.mem_get_info()[0]
    made = [LearnedProposal(ModelL96(dim=40), 0.05, 128, 1) for _ in range(8)]
    used = free0 - torch.cuda.mem_get_info()[0]
    for p in made:
        p.close()
    assert used <= 8 * (4 << 20), used


def test_long_traces_are_whole_and_take_no_memory(cuda):
    """At a learning rate far below every parameter's rounding (a zero weight
    moves to 1e-30) a step's loss depends on its minibatch alone, and minibatches follow the count of steps: the trace
    of one long call equals those of shorter ones, across the read-backs of
    1024 steps.  A call's device memory does not grow with its steps (300 000
    losses would take 2.4 MB)."""
    import torch
    from libbi_b200 import LearnedProposal, ModelL96

    data = _data(500, 11)

    def made():
        p = LearnedProposal(ModelL96(dim=40), 0.05, 128, 5)
        p.set_data(*data)
        return p

    p, q = made(), made()
    got = p.train(2600, 16, 1e-30)
    want = np.concatenate([q.train(n, 16, 1e-30) for n in (1, 1023, 1024, 552)])
    assert np.isfinite(got).all()
    np.testing.assert_array_equal(got, want)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    p.train(300000, 1, 1e-30)
    assert free0 - torch.cuda.mem_get_info()[0] < 1 << 20
    p.close()
    q.close()


def test_data_that_do_not_fit_leave_nothing_to_train_on(cuda):
    """A data set too large for the device's memory is refused, and training
    is refused after it (the rows of the one before are gone)."""
    from libbi_b200 import LearnedProposal, ModelL96
    from libbi_b200 import _native as N

    p = LearnedProposal(ModelL96(dim=40), 0.05, 128, 5)
    data = _data(200, 13)
    p.set_data(*data)
    ptrs = [t.data_ptr() for t in data]
    assert N.lib().bpf_proposal_set_data(p.handle, *ptrs, 2**31 - 1) == N.BPF_E_NOMEM  # 344 GB of means
    assert N.lib().bpf_proposal_train(p.handle, 1, 64, 1e-3, None) == N.BPF_E_INVALID
    p.set_data(*data)
    assert np.isfinite(p.train(2, 64, 1e-3)).all()
    p.close()
