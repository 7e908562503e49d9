"""A builder matrix of NaNs (mu so large that exp(dt mu) overflows): every index the factorisations and
the inverse form stays inside the matrix, the chain's status reaches the caller as HQ_E_NUMERIC, and
a healthy chain that lies behind it in the same context gives the bits it gives alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UP, DOWN = 0, 1


# one pivot panel and several, a ragged last panel, row slots 1 .. 8, G beyond one SM (13 .. 16); a single
# site is left out: its infinite scale leaves the builder matrix finite (G = 0, the limit)
@pytest.mark.parametrize("L", [2, 3, 4, 6, 8, 9, 11, 12, 13, 14, 15, 16])
def test_nan_builder_matrix(hq, L):
    good = dict(nl=L, u=4.0, mu=0.1, beta=0.6, nt=6, stabilization_pace=4, seed=3)
    modes = [hq.SWEEP_LAUNCHES] + ([hq.SWEEP_PERSISTENT] if L <= 12 else [])
    for mode in modes:
        alone, both = hq.Engine([good]), hq.Engine([dict(good, mu=1e6, seed=4), good])
        for e in (alone, both):
            if L <= 12:
                e.set_sweep_mode(mode)
            e.fields_random()
            e.init()
        with pytest.raises(hq.HqError) as ei:
            both.wrap_errors(0)
        assert ei.value.code == hq.capi.HQ_E_NUMERIC
        for e in (alone, both):
            e.sweep(UP, hq.SWEEP_MEASURE)
            e.sweep(DOWN, hq.SWEEP_MEASURE)
            e.sync()
        assert np.array_equal(alone.g(0), both.g(1)) and np.isfinite(both.g(1)).all()
        assert np.array_equal(alone.fields(0), both.fields(1))
        assert np.array_equal(alone.wrap_errors(0), both.wrap_errors(1))
        alone.close()
        both.close()


@pytest.mark.parametrize("L", [1, 4, 7, 8])
def test_nan_builder_matrix_noalloc(hq, L):
    import torch
    N = L * L
    f = torch.ones(6 * N, dtype=torch.int8, device="cuda")
    out = []
    for mu in (0.1, 1e6, 0.1):
        g = torch.zeros(N, N, dtype=torch.float64, device="cuda")
        rc = hq.lib().hq_equaltime_g_noalloc(L, 1.0, 4.0, mu, 0.6, 6, 4, f.data_ptr(), g.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream)
        assert rc == 0, hq.capi.last_error()
        out.append(g.cpu().numpy())
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[2])
