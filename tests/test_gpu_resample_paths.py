"""The resampler's kernels at the sizes where their splits change, on
log-weights that stress them, against the oracle: ancestors equal as whole
numbers (each is a function of exact sums of the same fixed-point weights, or
of the same comparisons, so nothing is left to a tolerance)."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = ("systematic", "multinomial", "metropolis")
B = 5


def _patterns(n, seed):
    """Log-weights with maximum 0: spread ones; one particle with nearly all
    the weight (its copies are written by a whole block); many without
    weight (-inf, NaN and far below the largest)."""
    rng = np.random.default_rng(seed)
    z = 2.0 * rng.standard_normal(n)
    spread = z - z.max()
    one = np.full(n, -60.0) + 0.5 * rng.random(n)
    one[rng.integers(n)] = 0.0
    few = spread.copy()
    u = rng.random(n)
    few[u < 0.3] = -np.inf
    few[(u >= 0.3) & (u < 0.4)] = np.nan
    few[(u >= 0.4) & (u < 0.6)] = -1.0e4
    few[rng.integers(n)] = 0.0
    return {"spread": spread, "one": one, "few": few}


def _want(oracle, kind, lw, uniforms):
    """(ancestors in the order of the draws or sorted, permuted ancestors)"""
    if kind == "systematic":
        return oracle.systematic(lw, uniforms[0], permute=False)[3], oracle.systematic(lw, uniforms[0], permute=True)[3]
    if kind == "multinomial":
        a = oracle.multinomial(lw, uniforms, 0)[1]
    else:
        a = oracle.metropolis(lw, B, uniforms, 0)[1]
    return a, oracle.permute_rule(a)


def _own_uniforms(oracle, kind, n, seed, step):
    return oracle.resample_uniforms(KINDS.index(kind), n, B, seed, step)


@pytest.mark.parametrize("max_n", [4096, 8192, 16384, 32768])
def test_batch_resampler_at_cluster_and_run_edges(cuda, oracle, max_n):
    """Every kind at sizes around the runs of 16, the thread counts and the
    CTAs' shares, with every cluster size that holds the largest filter (1 to
    8 CTAs; small filters leave CTAs of their cluster empty) and every thread
    count."""
    import torch
    from libbi_b200 import BatchedBootstrapPF, ModelPZ
    from libbi_b200 import _native as N

    sizes = [2, 15, 17, 128, 129, 513, 1024, 4095, max_n - 1, max_n]
    ns = [n for n in sizes for _ in KINDS]
    kinds = list(KINDS) * len(sizes)
    seeds = [70 + f for f in range(len(ns))]
    batch = BatchedBootstrapPF([ModelPZ()] * len(ns), ns, kinds, seeds, ess_rel=1.0, metropolis_steps=B)
    y = torch.full((len(ns), 1), 0.5, dtype=torch.float64, device="cuda")
    clusters = [g for g in (1, 2, 4, 8) if max_n <= 4096 * g]
    for ctas in {1, 2, 3, 4, 16} - set(clusters):
        with pytest.raises(N.BpfError):
            batch.resample_cluster(ctas)
    for i, (ctas, threads) in enumerate(itertools.product(clusters, (256, 512, 1024))):
        pattern = ("spread", "one", "few")[(i + i // 3) % 3]
        assert batch.resample_cluster(ctas) == ctas
        batch.resample_threads(threads)
        batch.init()
        batch.step_device(0.0, 1.0, y)
        torch.cuda.synchronize()
        _, lw, anc, offs = batch.state()
        given = []
        host = lw.cpu().numpy()
        for f, n in enumerate(ns):
            # the gate and the largest log-weight are the step's own
            given.append(host[offs[f]:offs[f] + n].max() + _patterns(n, f)[pattern])
            lw[offs[f]:offs[f] + n] = torch.as_tensor(given[f], device="cuda")
        torch.cuda.synchronize()
        batch.step_device(1.0, 2.0, y)
        torch.cuda.synchronize()
        got = anc.cpu().numpy()
        for f, n in enumerate(ns):
            want = _want(oracle, kinds[f], given[f], _own_uniforms(oracle, kinds[f], n, seeds[f], 2))[1]
            np.testing.assert_array_equal(got[offs[f]:offs[f] + n], want, err_msg=f"{kinds[f]} {n} {pattern} {ctas} {threads}")
    batch.close()


@pytest.mark.parametrize("kind,n", [("systematic", 2), ("systematic", 8192), ("systematic", 8193),
                                    ("multinomial", 32768), ("multinomial", 32769),
                                    ("metropolis", 4096), ("metropolis", 4097)])
def test_single_filter_on_both_sides_of_the_cluster_limit(cuda, oracle, kind, n):
    """The largest filter that one cluster resamples and the next one, which
    the grid-wide kernels do: the same rule gives both their ancestors."""
    import torch
    from libbi_b200 import BootstrapPF, ModelPZ

    pf = BootstrapPF(ModelPZ(), n, resampler=kind, ess_rel=1.0, seed=9, metropolis_steps=B)
    for pattern in ("spread", "one", "few"):
        pf.init()
        pf.step(0.0, 1.0, 0.5)
        _, lw, anc = pf.state()
        given = lw.cpu().numpy().max() + _patterns(n, n)[pattern]
        lw[:] = torch.as_tensor(given, device="cuda")
        torch.cuda.synchronize()
        assert pf.step(1.0, 2.0, 0.5).resampled
        want = _want(oracle, kind, given, _own_uniforms(oracle, kind, n, 9, 2))[1]
        np.testing.assert_array_equal(anc.cpu().numpy(), want, err_msg=pattern)
    pf.close()


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 33, 2047, 2049, 65537, 300001])
def test_stand_alone_resamplers_on_stressed_weights(cuda, oracle, n, offset):
    """The maximum-only first pass (16-byte loads when the log-weights allow
    them: offset 0; one value at a time otherwise), the block-wide searches
    and the Metropolis comparisons, sorted and permuted."""
    import torch
    from libbi_b200 import MetropolisResampler, MultinomialResampler, SystematicResampler

    made = {"systematic": SystematicResampler(max_n=n), "multinomial": MultinomialResampler(max_n=n),
            "metropolis": MetropolisResampler(max_n=n, B=B)}
    rng = np.random.default_rng(n)
    for pattern, lw in _patterns(n, n).items():
        lw = lw - 700.0
        buf = torch.empty(n + offset, dtype=torch.float64, device="cuda")
        lw_d = buf[offset:]
        lw_d.copy_(torch.as_tensor(lw, device="cuda"))
        for kind, r in made.items():
            u = rng.random({"systematic": 1, "multinomial": n, "metropolis": 2 * n * B}[kind])
            u_d = torch.as_tensor(u, device="cuda")
            plain, permuted = _want(oracle, kind, lw, u)
            got = r.ancestors(lw_d, u_d, permute=False).cpu().numpy()
            np.testing.assert_array_equal(got, plain, err_msg=f"{kind} {pattern}")
            got = r.ancestors(lw_d, u_d, permute=True).cpu().numpy()
            np.testing.assert_array_equal(got, permuted, err_msg=f"{kind} {pattern} permuted")
    for r in made.values():
        r.close()


WIDE = 148 * 8 * 256  # slots that one block per 256 of them still holds at once


@pytest.mark.parametrize("n", [2**18 - 1, 2**18, WIDE, WIDE + 1, 2**19 - 1, 2**19, 1000003])
def test_stand_alone_resamplers_at_their_wide_forms(cuda, oracle, n):
    """Both sides of the sizes from which a multinomial tile holds 4 and 8
    particles per thread and a thread searches for four slots, and an odd size
    well beyond them: the multinomial ancestors sorted and permuted, the
    systematic ones sorted (permuted they take another kernel), the Metropolis
    ones permuted (unpermuted ones need no search)."""
    import torch
    from libbi_b200 import MetropolisResampler, MultinomialResampler, SystematicResampler

    made = {"multinomial": (MultinomialResampler(max_n=n), (False, True)),
            "systematic": (SystematicResampler(max_n=n), (False,)),
            "metropolis": (MetropolisResampler(max_n=n, B=B), (True,))}
    rng = np.random.default_rng(n)
    for pattern, lw in _patterns(n, n).items():
        lw_d = torch.as_tensor(lw, device="cuda")
        for kind, (r, forms) in made.items():
            u = rng.random({"systematic": 1, "multinomial": n, "metropolis": 2 * n * B}[kind])
            u_d = torch.as_tensor(u, device="cuda")
            want = _want(oracle, kind, lw, u)
            for permute in forms:
                got = r.ancestors(lw_d, u_d, permute=permute).cpu().numpy()
                np.testing.assert_array_equal(got, want[permute], err_msg=f"{kind} {pattern} permute={permute}")
    for r, _ in made.values():
        r.close()


@pytest.mark.parametrize("n,s", [(100003, 16), (100003, 17), (400003, 4), (400003, 5)])
def test_childless_slots_spread_thinly(cuda, oracle, n, s):
    """Every s-th particle takes its neighbour as ancestor, so a block's 256
    ranks (1024 with four searches per thread) are bracketed by 255 s (1023 s)
    particles: just within and just beyond the 4096 that the fill of the
    childless slots keeps in shared memory."""
    import torch
    from libbi_b200 import MetropolisResampler

    lw = np.zeros(n)
    target = np.arange(n)
    target[: n - 1: s] += 1
    u = np.empty(2 * n)
    u[0::2] = (target + 0.5) / n  # the proposed ancestor
    u[1::2] = 0.5  # accepted: log u < 0
    r = MetropolisResampler(max_n=n, B=1)
    plain = oracle.metropolis(lw, 1, u, 0)[1]
    np.testing.assert_array_equal(plain, target)
    got = r.ancestors(torch.as_tensor(lw, device="cuda"), torch.as_tensor(u, device="cuda"), permute=True)
    np.testing.assert_array_equal(got.cpu().numpy(), oracle.permute_rule(plain))
    r.close()
