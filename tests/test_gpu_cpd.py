"""GPU CP-ALS against the oracle and the reference's recorded fits.

Factors are float32 on the device (MTTKRP accumulates in float32, Grams /
Cholesky / fit in float64), so the bound is relative: |fit - fit_ref| <=
1e-5 * fit_ref per iteration, and the final factors within 1e-3
(normwise) of the FP64 oracle."""
import numpy as np
import pytest

import alto_b200 as A
import oracle as O
from alto_b200 import synth
from conftest import load_fixture

pytestmark = pytest.mark.gpu


def init_model(dims, R, seed):
    init = synth.init_values(int(np.sum(dims)) * R, seed=seed)
    U0, off = [], 0
    for d in dims:
        U0.append(init[off:off + int(d) * R].reshape(int(d), R).copy())
        off += int(d) * R
    return U0


def test_med_fits_match_reference(golden):
    g = golden["cpd_als_med"]
    dims, cidx, vals = load_fixture("med")
    R = g["rank"]
    U0 = init_model(dims, R, g["init_seed"])
    t = A.create_alto(dims, cidx, vals)
    U, lam, fits, it = A.cpd_alto(t, U0, np.ones(R), R, 8, 1e-12)
    assert it == g["iters"]
    np.testing.assert_allclose(fits, g["fits"], rtol=1e-5)


@pytest.mark.parametrize("R,fit_mode", [(8, A.FIT_REFERENCE), (16, A.FIT_EXACT), (32, A.FIT_REFERENCE)])
def test_random_against_oracle(R, fit_mode):
    dims = np.array([60, 70, 80], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 20000, seed=R)
    vals = vals.astype(np.float32).astype(np.float64)
    U0 = [u.astype(np.float32).astype(np.float64) for u in init_model(dims, R, R)]
    t = A.create_alto(dims, cidx, vals)
    U, lam, fits, it = A.cpd_alto(t, U0, np.ones(R), R, 6, 1e-12, fit_mode=fit_mode)
    Uo, lo, fo, ito = O.cpd_als(O.build(dims, cidx, vals), U0, np.ones(R), R, 6, 1e-12,
                                fit_exact=fit_mode == A.FIT_EXACT)
    assert it == ito == 6
    np.testing.assert_allclose(fits, fo, rtol=1e-5)
    for a, b in zip(U, Uo):
        assert np.abs(a - b).max() <= 1e-3 * np.abs(b).max()
    np.testing.assert_allclose(lam, lo, rtol=1e-3)


def test_five_modes_and_bf16_storage():
    dims = np.array([500, 400, 300, 50, 20], np.uint64)
    cidx, vals = synth.powerlaw_coo(dims, 60000, [1.1, 1.1, None, None, None], seed=2)
    R = 16
    U0 = init_model(dims, R, 1)
    t = A.create_alto(dims, cidx, vals)
    _, _, f32, _ = A.cpd_alto(t, U0, np.ones(R), R, 5, 1e-12, storage=A.F32)
    _, _, fb, _ = A.cpd_alto(t, U0, np.ones(R), R, 5, 1e-12, storage=A.BF16)
    _, _, fo, _ = O.cpd_als(O.build(dims, cidx, vals), U0, np.ones(R), R, 5, 1e-12)
    np.testing.assert_allclose(f32, fo, rtol=1e-4)
    np.testing.assert_allclose(fb, fo, rtol=5e-3)


def test_early_stop_matches_epsilon():
    dims = np.array([40, 50, 60], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 8000, seed=5)
    vals = vals.astype(np.float32).astype(np.float64)
    R = 8
    U0 = [u.astype(np.float32).astype(np.float64) for u in init_model(dims, R, 2)]
    t = A.create_alto(dims, cidx, vals)
    _, _, fits, it = A.cpd_alto(t, U0, np.ones(R), R, 50, 1e-3)
    _, _, fo, ito = O.cpd_als(O.build(dims, cidx, vals), U0, np.ones(R), R, 50, 1e-3)
    assert it == ito


@pytest.mark.parametrize("R", [1, 7, 9, 15, 17, 31, 33, 48, 63, 64, 65, 100])
def test_ranks_around_the_column_tiles(R):
    """Every width of the row solves, the set-up and the Grams; the module's
    bound on fits is relative, so the data have a fit of about one half."""
    rng = np.random.default_rng(R)
    dims = np.array([150, 131, 160], np.uint64)
    cidx = np.stack([rng.integers(0, int(d), 30000) for d in dims])
    cidx = np.unique(cidx, axis=1).astype(np.uint64)
    vals = (1.0 + rng.uniform(0, 1, cidx.shape[1])).astype(np.float32).astype(np.float64)
    U0 = [u.astype(np.float32).astype(np.float64) for u in init_model(dims, R, R)]
    t = A.create_alto(dims, cidx, vals)
    U, lam, fits, it = A.cpd_alto(t, U0, np.ones(R), R, 4, 1e-12)
    _, lo, fo, ito = O.cpd_als(O.build(dims, cidx, vals), U0, np.ones(R), R, 4, 1e-12)
    assert it == ito
    # a float32 MTTKRP is right to 1e-6; the fit is 1 - sqrt(y) with an error of y below 4e-6
    np.testing.assert_allclose(fits, fo, rtol=0, atol=1e-5)


def test_more_iterations_than_a_window_of_fits():
    """Without a stopping test the fits are read back 64 at a time."""
    dims = np.array([40, 50, 60], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 8000, seed=6)
    vals = vals.astype(np.float32).astype(np.float64)
    R = 2
    U0 = [u.astype(np.float32).astype(np.float64) for u in init_model(dims, R, 3)]
    t = A.create_alto(dims, cidx, vals)
    _, _, fits, it = A.cpd_alto(t, U0, np.ones(R), R, 131, 0.0)
    _, _, fo, ito = O.cpd_als(O.build(dims, cidx, vals), U0, np.ones(R), R, 131, 0.0)
    assert it == ito == 131 and len(fits) == 131
    # the bound of a single fit, in absolute terms, over the two factors' whole descent
    np.testing.assert_allclose(fits, fo, rtol=0, atol=1e-4)


@pytest.mark.parametrize("heavy", [4000, 4096, 4097, 8191, 8192, 8193, 20000])
@pytest.mark.parametrize("nmodes", [3, 4, 5])
def test_a_row_with_a_long_run(nmodes, heavy):
    """One row of mode 0 holds `heavy` nonzeros: found for certain from 8192 on
    (then that mode's walk is reproducible), right on either side."""
    rng = np.random.default_rng(heavy + nmodes)
    dims = np.array([60, 170, 150, 20, 10][:nmodes], np.uint64)
    flat = rng.choice(170 * 150, heavy, replace=False)
    rest = np.arange(170 * 59)
    c = np.concatenate([np.stack([np.zeros(heavy, np.int64), flat % 170, flat // 170]),
                        np.stack([1 + rest // 170, rest % 170, rng.integers(0, 150, rest.size)])], axis=1)
    c = np.concatenate([c, np.stack([rng.integers(0, int(d), c.shape[1]) for d in dims[3:]])]) if nmodes > 3 else c
    c = c.astype(np.uint64)
    vals = (1.0 + rng.uniform(0, 1, c.shape[1])).astype(np.float32).astype(np.float64)
    R = 8
    U0 = [u.astype(np.float32).astype(np.float64) for u in init_model(dims, R, 3)]
    t = A.create_alto(dims, c, vals)
    U, lam, fits, it = A.cpd_alto(t, U0, np.ones(R), R, 4, 0.0)
    _, _, fo, _ = O.cpd_als(O.build(dims, c, vals), U0, np.ones(R), R, 4, 0.0)
    np.testing.assert_allclose(fits, fo, rtol=0, atol=1e-5)


@pytest.mark.parametrize("spare", [256, 560])
def test_copies_that_do_not_fit(spare):
    """With `spare` MiB of device memory left, none or one of the modes' row-sorted
    copies (256 MB each) fits beside the call's own 160 MB: the other modes are
    walked without, and the fits are those of a run with every copy, to the
    module's bound on a single fit in absolute terms."""
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    dims, nnz, R = np.array([200000, 150000, 100000], np.uint64), 16000000, 16
    idx = [torch.randint(0, int(d), (nnz,), generator=g, device="cuda") for d in dims]
    vals = torch.rand(nnz, generator=g, device="cuda") + 0.5
    U0 = init_model(dims, R, 4)
    t = A.create_alto(dims, idx, vals)
    _, _, want, _ = A.cpd_alto(t, U0, np.ones(R), R, 4, 0.0)
    t.close()
    t = A.create_alto(dims, idx, vals)
    before = t.device_bytes()
    A.release_memory()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (spare << 20), dtype=torch.uint8, device="cuda")
    try:
        _, _, fits, _ = A.cpd_alto(t, U0, np.ones(R), R, 4, 0.0)
    finally:
        del filler
        torch.cuda.empty_cache()
    copies = (t.device_bytes() - before) / (16 * nnz)
    assert 0 <= copies < (0.5 if spare == 256 else 2.5)
    np.testing.assert_allclose(fits, want, rtol=0, atol=1e-5)
    _, _, fits, _ = A.cpd_alto(t, U0, np.ones(R), R, 4, 0.0)  # with room again
    np.testing.assert_allclose(fits, want, rtol=0, atol=1e-5)
    assert (t.device_bytes() - before) / (16 * nnz) > 2.9


def test_room_for_factors_and_staging():
    """A call needs the factors, the MTTKRP's output and one float64 factor of device
    memory (256 + 256 + 512 MiB here), and no fourth array of a factor's size."""
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    dims, nnz, R = np.array([1 << 21, 64, 64], np.uint64), 100000, 32
    idx = [torch.randint(0, int(d), (nnz,), generator=g, device="cuda") for d in dims]
    t = A.create_alto(dims, idx, torch.rand(nnz, generator=g, device="cuda") + 0.5)
    U0 = init_model(dims, R, 4)
    _, _, want, _ = A.cpd_alto(t, U0, np.ones(R), R, 2, 0.0)
    A.release_memory()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (1150 << 20), dtype=torch.uint8, device="cuda")
    try:
        _, _, fits, _ = A.cpd_alto(t, U0, np.ones(R), R, 2, 0.0)
    finally:
        del filler
        torch.cuda.empty_cache()
    np.testing.assert_allclose(fits, want, rtol=0, atol=1e-5)
