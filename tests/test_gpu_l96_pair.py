"""The Lorenz '96 transition's two forms (one or two threads per particle) on
both sides of the sizes where the choice changes, single and batched, against
the oracle's filter: states equal, log-weights to the rounding of the sums'
order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BLOCK = 128  # particles of a transition block
CASES = [(dim, prec, n) for dim in (8, 16, 32, 40) for prec in ("f32", "f64") for n in (1, BLOCK + 1)]
CASES += [(4, "f64", BLOCK + 1)]
CASES += [(40, "f32", 2 * 148 * BLOCK + i) for i in (0, 1)] + [(40, "f32", 3 * 148 * BLOCK + i) for i in (0, 1)]
CASES += [(40, "f64", 2 * 148 * BLOCK + 1)]
CASES += [(dim, "f64", 2 * 148 * BLOCK + i) for dim in (8, 16) for i in (0, 1)]


def _want(oracle, model, n, seed, y, T, dt):
    from libbi_b200 import _native as N

    cfg = N.Config()
    cfg.nparticles = n
    cfg.resampler = N.BPF_RESAMPLER_SYSTEMATIC
    cfg.ess_rel = 0.5
    cfg.seed = seed
    return oracle.filter(model.desc(), cfg, np.ascontiguousarray(y), T, 0.0, dt)


@pytest.mark.parametrize("dim,prec,n", CASES)
def test_transition_forms_match_oracle(cuda, oracle, dim, prec, n):
    from libbi_b200 import BootstrapPF, ModelL96

    model, T, dt, seed = ModelL96(dim=dim, precision=prec), 3, 0.05, 17
    y = oracle.simulate(model.desc(), 3, T, 0.0, dt)[0]
    want = _want(oracle, model, n, seed, y, T, dt)
    assert want["rc"] == 0
    pf = BootstrapPF(model, n, ess_rel=0.5, seed=seed)
    for _ in range(2):  # the second run replays the first one's graph
        ll, inc, ess = pf.filter(y, 0.0, dt)
    x, lw, _ = pf.state()
    np.testing.assert_array_equal(x.cpu().numpy()[:, :n], want["x"][:, :n])
    np.testing.assert_allclose(lw.cpu().numpy(), want["lw"], rtol=1e-12)
    np.testing.assert_allclose(inc, want["inc"], rtol=1e-10, atol=1e-9)
    np.testing.assert_allclose(ess, want["ess"], rtol=1e-9)
    pf.close()


@pytest.mark.parametrize("total", [2 * 148, 2 * 148 + 1, 3 * 148, 3 * 148 + 1])
def test_batched_forms_match_oracle(cuda, oracle, total):
    """Batches of `total` transition blocks: two filters of whole blocks and
    one of a single block that is not full."""
    from libbi_b200 import BatchedBootstrapPF, ModelL96

    nb = (total - 1) // 2
    ns = [min(nb * BLOCK, 32768), BLOCK - 1, min(nb * BLOCK, 32768)]
    while sum((n + BLOCK - 1) // BLOCK for n in ns) < total:
        ns.append(min(32768, BLOCK * (total - sum((n + BLOCK - 1) // BLOCK for n in ns))))
    model, T, dt = ModelL96(dim=40), 2, 0.05
    y = oracle.simulate(model.desc(), 5, T, 0.0, dt)[0]
    seeds = [30 + f for f in range(len(ns))]
    batch = BatchedBootstrapPF([model] * len(ns), ns, ["systematic"] * len(ns), seeds, ess_rel=0.5)
    _, inc, _, st = batch.filter(np.repeat(y[:, None], len(ns), axis=1), 0.0, dt)
    assert (st == 0).all()
    x, lw, _, offs = batch.state()
    x, lw = x.cpu().numpy(), lw.cpu().numpy()
    for f, n in enumerate(ns):
        want = _want(oracle, model, n, seeds[f], y, T, dt)
        np.testing.assert_array_equal(x[:, offs[f]:offs[f] + n], want["x"][:, :n])
        np.testing.assert_allclose(lw[offs[f]:offs[f] + n], want["lw"], rtol=1e-12)
        np.testing.assert_allclose(inc[:, f], want["inc"], rtol=1e-10, atol=1e-9)
    batch.close()
