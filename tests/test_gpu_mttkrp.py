"""GPU MTTKRP against the FP64 oracle.

The oracle receives the factor values the GPU reads (float32, or bfloat16
for the BF16 path, widened to float64), so the comparison isolates the
float32 accumulation.  Bound: max |gpu - oracle| / max |oracle| <= 1e-5
(normwise) for every mode, rank and variant."""
import numpy as np
import pytest

import alto_b200 as A
import oracle as O
from alto_b200 import synth
from conftest import FIXTURE_NAMES, load_fixture

pytestmark = pytest.mark.gpu
TOL = 1e-5
ALL_VARIANTS = (A.AUTO, A.ATOMIC, A.STAGED, A.SORTED, A.ATOMIC | A.FEED_BULK, A.SORTED | A.FEED_BULK)
# the row-sorted walks that exist for 3-mode tensors only
THREE_MODE_FEEDS = (A.SORTED | A.FEED_DENSE, A.SORTED | A.FEED_FIXED_TARGET)


def to_dev(F, dtype):
    import torch

    return [torch.tensor(f, dtype=torch.float32, device="cuda").to(dtype).contiguous() for f in F]


def seen_by_gpu(Fd):
    return [f.float().cpu().numpy().astype(np.float64) for f in Fd]


def rel_err(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def check_modes(dims, cidx, vals, R, variants=(A.AUTO,), dtype=None, seed=0):
    import torch

    dtype = dtype or torch.float32
    rng = np.random.default_rng(seed)
    F = [rng.uniform(-1.0, 1.0, (int(d), R)) for d in dims]
    Fd = to_dev(F, dtype)
    Fo = seen_by_gpu(Fd)
    t = A.create_alto(dims, cidx, vals)
    vals32 = vals.astype(np.float32).astype(np.float64)
    enc = O.build(dims, cidx, vals32)
    for m in range(len(dims)):
        fs = [f.copy() for f in Fo]
        fs[m][:] = 0
        ref = O.mttkrp(enc, m, fs, R)[m]
        extra = THREE_MODE_FEEDS if len(dims) == 3 and A.SORTED in variants else ()
        for v in tuple(variants) + extra:
            out = t.mttkrp(m, Fd, R, variant=v).cpu().numpy()
            assert rel_err(out, ref) <= TOL, (m, v, rel_err(out, ref))


@pytest.mark.parametrize("name", FIXTURE_NAMES)
def test_fixtures_rank8(name):
    dims, cidx, vals = load_fixture(name)
    check_modes(dims, cidx, vals, 8, variants=ALL_VARIANTS)


@pytest.mark.parametrize("R", [4, 8, 16, 32, 64, 128, 10, 33])
def test_uniform_ranks(R):
    dims = np.array([1000, 1000, 1000], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 150000, seed=R)
    check_modes(dims, cidx, vals, R, variants=ALL_VARIANTS, seed=R)


@pytest.mark.parametrize("R", [8, 16, 32, 64])
def test_bf16_factor_storage(R):
    import torch

    dims = np.array([800, 700, 900], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 100000, seed=R + 1)
    check_modes(dims, cidx, vals, R, variants=(A.AUTO, A.ATOMIC, A.SORTED, A.SORTED | A.FEED_BULK), dtype=torch.bfloat16, seed=R)


def test_power_law_128bit_keys():
    """Zipf-1.2 coordinates with scattered labels and a 65-bit key."""
    dims = np.array([4800000, 1800000, 1800000], np.uint64)
    cidx, vals = synth.powerlaw_coo(dims, 200000, [1.2, 1.2, 1.2], seed=3, values="lognormal")
    check_modes(dims, cidx, vals, 32, variants=ALL_VARIANTS)


def test_five_modes_rank64():
    dims = np.array([100000, 100000, 10000, 1000, 100], np.uint64)
    cidx, vals = synth.powerlaw_coo(dims, 150000, [1.1, 1.1, None, None, None], seed=4)
    check_modes(dims, cidx, vals, 64, variants=ALL_VARIANTS)


def test_stream_mode_single_row():
    dims = np.array([1, 3000, 4000, 500], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 100000, seed=6)
    import torch

    R = 16
    rng = np.random.default_rng(1)
    F = [rng.uniform(-1, 1, (int(d), R)) for d in dims]
    Fd = to_dev(F, torch.float32)
    t = A.init_salto(dims, cidx, vals, 1, stream_mode=0)
    assert t.choose_variant(0, R) == A.STREAM
    enc = O.build(dims, cidx, vals.astype(np.float32).astype(np.float64))
    fs = seen_by_gpu(Fd)
    fs[0][:] = 0
    ref = O.mttkrp(enc, 0, fs, R)[0]
    out = t.mttkrp(0, Fd, R).cpu().numpy()
    assert rel_err(out, ref) <= TOL


def test_accumulate_semantics():
    import torch

    dims = np.array([300, 200, 100], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 30000, seed=8)
    R = 16
    rng = np.random.default_rng(2)
    F = [rng.uniform(-1, 1, (int(d), R)) for d in dims]
    Fd = to_dev(F, torch.float32)
    t = A.create_alto(dims, cidx, vals)
    base = Fd[1].clone()
    A.mttkrp_alto_par(1, Fd, R, t)  # accumulates into Fd[1]
    fresh = t.mttkrp(1, Fd, R).cpu().numpy()
    np.testing.assert_allclose(Fd[1].cpu().numpy(), base.cpu().numpy() + fresh, rtol=1e-5, atol=1e-5)


def test_host_buffer_entry_point():
    dims = np.array([400, 500, 600], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 50000, seed=10)
    R = 16
    rng = np.random.default_rng(3)
    F = [rng.uniform(-1, 1, (int(d), R)) for d in dims]
    t = A.create_alto(dims, cidx, vals)
    for m in range(3):
        fs = [f.copy() for f in F]
        start = fs[m].copy()
        t.mttkrp_host(m, fs, R)
        fo = [f.astype(np.float32).astype(np.float64) for f in F]
        fo[m][:] = 0
        ref = O.mttkrp(O.build(dims, cidx, vals.astype(np.float32).astype(np.float64)), m, fo, R)[m]
        assert rel_err(fs[m] - start, ref) <= TOL


def test_host_buffer_changed_mask_matches_full_copies():
    """A CP-ALS-like sequence of host-buffer MTTKRPs in which the caller
    rewrites the factor it just received (here: halves it) before the next
    call and declares only that factor changed (alto_mttkrp_host_changed):
    every call still matches the oracle on the caller's current arrays
    (a stale device copy would be off by the halving)."""
    dims = np.array([400, 500, 600], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 50000, seed=12)
    R = 16
    rng = np.random.default_rng(4)
    G = [rng.uniform(-1, 1, (int(d), R)) for d in dims]
    t = A.create_alto(dims, cidx, vals)
    enc = O.build(dims, cidx, vals.astype(np.float32).astype(np.float64))
    prev = None
    for it in range(2):
        for m in range(3):
            start = G[m].copy()
            fo = [g.astype(np.float32).astype(np.float64) for g in G]
            fo[m][:] = 0
            ref = O.mttkrp(enc, m, fo, R)[m]
            t.mttkrp_host(m, G, R, changed=range(3) if prev is None else [prev])
            assert rel_err(G[m] - start, ref) <= TOL, (it, m)
            G[m] *= 0.5
            prev = m
    t.close()


def test_launch_counter_advances():
    import torch

    dims = np.array([50, 60, 70], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 1000, seed=1)
    t = A.create_alto(dims, cidx, vals)
    Fd = to_dev([np.ones((int(d), 8)) for d in dims], torch.float32)
    n0 = A.kernel_launches()
    t.mttkrp(0, Fd, 8)
    torch.cuda.synchronize()
    assert A.kernel_launches() > n0


def test_autotune_records_a_choice_per_mode():
    import torch

    dims = np.array([4800000, 1800000, 1800000], np.uint64)
    cidx, vals = synth.powerlaw_coo(dims, 300000, [1.2, 1.2, 1.2], seed=5, values="lognormal")
    R = 32
    rng = np.random.default_rng(4)
    Fd = to_dev([rng.uniform(-1, 1, (int(d), R)) for d in dims], torch.float32)
    t = A.create_alto(dims, cidx, vals)
    chosen = t.autotune(Fd, R)
    assert len(chosen) == 3 and all(c in (A.ATOMIC, A.STAGED, A.SORTED) for c in chosen)
    for m in range(3):
        assert t.choose_variant(m, R) == chosen[m]
    Fo = seen_by_gpu(Fd)
    enc = O.build(dims, cidx, vals.astype(np.float32).astype(np.float64))
    for m in range(3):
        fs = [f.copy() for f in Fo]
        fs[m][:] = 0
        ref = O.mttkrp(enc, m, fs, R)[m]
        assert rel_err(t.mttkrp(m, Fd, R).cpu().numpy(), ref) <= TOL


# ------------------------------------------------- row-sorted and any-rank walks

@pytest.mark.parametrize("R", [1, 3, 6, 10, 12, 24, 33, 64, 100, 130, 260])
@pytest.mark.parametrize("nmodes", [2, 3, 4, 5, 6])
def test_walks_of_every_rank_and_mode_count(nmodes, R):
    """The row-sorted and the any-rank walk at ranks around their lane splits
    (one lane, a lane group that does not divide the warp, several column
    windows) and with factors and output at odd addresses: the same bound as
    the specialised kernels.  The last run's length leaves partial steps."""
    import torch

    dims = np.array([37, 53, 41, 29, 31, 23][:nmodes], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 1501 if nmodes == 2 else 9973, seed=R)
    t = A.create_alto(dims, cidx, vals)
    enc = O.build(dims, cidx, vals.astype(np.float32).astype(np.float64))
    rng = np.random.default_rng(R)
    F = [rng.uniform(-1.0, 1.0, (int(d), R)) for d in dims]
    for dtype in (torch.float32, torch.bfloat16):
        for shift in (0, 1, 2):
            Fd = []
            for f in F:
                room = torch.zeros(f.size + shift, dtype=dtype, device="cuda")
                room[shift:] = torch.tensor(f.ravel(), dtype=torch.float32, device="cuda").to(dtype)
                Fd.append(room[shift:].view(f.shape))
            Fo = seen_by_gpu(Fd)
            for m in range(nmodes):
                fs = [f.copy() for f in Fo]
                fs[m][:] = 0
                ref = O.mttkrp(enc, m, fs, R)[m]
                room = torch.full((int(dims[m]) * R + shift,), np.nan, device="cuda")
                out = room[shift:].view(int(dims[m]), R)
                for v in (A.SORTED, A.ATOMIC, A.AUTO):
                    t.mttkrp(m, Fd, R, out=out, variant=v)
                    got = out.cpu().numpy()
                    assert rel_err(got, ref) <= TOL, (dtype, shift, m, v, rel_err(got, ref))
                    assert shift == 0 or bool(torch.isnan(room[:shift]).all())  # nothing written before it


def test_decoded_copies_of_keys_above_96_bits():
    dims = np.array([700000, 650000, 800000, 600000, 900000], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 30000, seed=3)
    check_modes(dims, cidx, vals, 8, variants=(A.SORTED, A.ATOMIC, A.SORTED | A.FEED_BULK))


# ------------------------------------------------- deterministic variant

def check_deterministic(dims, cidx, vals, R, seed=0, stream_mode=-1):
    """DETERMINISTIC against the oracle, and bit-identical on a second run
    with other MTTKRP work (atomic variants) launched in between."""
    import torch

    rng = np.random.default_rng(seed)
    Fd = to_dev([rng.uniform(-1.0, 1.0, (int(d), R)) for d in dims], torch.float32)
    Fo = seen_by_gpu(Fd)
    t = A.init_salto(dims, cidx, vals, 1, stream_mode=stream_mode) if stream_mode >= 0 else \
        A.create_alto(dims, cidx, vals)
    enc = O.build(dims, cidx, vals.astype(np.float32).astype(np.float64))
    for m in range(len(dims)):
        fs = [f.copy() for f in Fo]
        fs[m][:] = 0
        ref = O.mttkrp(enc, m, fs, R)[m]
        first = t.mttkrp(m, Fd, R, variant=A.DETERMINISTIC)
        assert rel_err(first.cpu().numpy(), ref) <= TOL, (m, rel_err(first.cpu().numpy(), ref))
        for v in (A.ATOMIC, A.SORTED):
            t.mttkrp(m, Fd, R, variant=v)
        again = t.mttkrp(m, Fd, R, variant=A.DETERMINISTIC)
        assert torch.equal(first, again), m


@pytest.mark.parametrize("name", FIXTURE_NAMES)
def test_deterministic_fixtures(name):
    dims, cidx, vals = load_fixture(name)
    check_deterministic(dims, cidx, vals, 8)


@pytest.mark.parametrize("R", [8, 16, 32, 64, 128])
def test_deterministic_ranks(R):
    dims = np.array([1000, 1000, 1000], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 150000, seed=R + 40)
    check_deterministic(dims, cidx, vals, R, seed=R)


def test_deterministic_hot_rows_and_128bit_keys():
    """Zipf 2.0: a few rows hold most nonzeros, so their runs span many
    lane-group sub-ranges (the long-chain fix-up)."""
    dims = np.array([4800000, 1800000, 1800000], np.uint64)
    cidx, vals = synth.powerlaw_coo(dims, 200000, [2.0, 1.2, 2.0], seed=13, values="lognormal")
    check_deterministic(dims, cidx, vals, 32)


def test_deterministic_five_modes_and_stream_row():
    dims = np.array([100000, 100000, 10000, 1000, 100], np.uint64)
    cidx, vals = synth.powerlaw_coo(dims, 150000, [1.1, 1.1, None, None, None], seed=14)
    check_deterministic(dims, cidx, vals, 64)
    dims = np.array([1, 3000, 4000, 500], np.uint64)  # every nonzero in one output row
    cidx, vals = synth.uniform_coo(dims, 100000, seed=15)
    check_deterministic(dims, cidx, vals, 16, stream_mode=0)


@pytest.mark.parametrize("R", [8, 32, 64, 128])
@pytest.mark.parametrize("nnz", [1, 63, 1000, 70001])
@pytest.mark.parametrize("dims", [[1, 40, 50], [1, 3, 2000, 9], [7, 90, 20, 11, 5]])
def test_deterministic_chunks(dims, nnz, R):
    """Chunk edges of the deterministic walk: a mode of one row (every slot one
    run), runs longer and shorter than a lane group's share, fewer nonzeros than
    lane groups, partial steps; the slots' rows are written once per call, also
    over an output that holds other values."""
    import torch

    dims = np.array(dims, np.uint64)
    nnz = int(min(nnz, np.prod(dims.astype(np.float64)) // 2))
    cidx, vals = synth.uniform_coo(dims, nnz, seed=R)
    check_deterministic(dims, cidx, vals, R, seed=R)
    t = A.create_alto(dims, cidx, vals)
    Fd = to_dev([np.ones((int(d), R)) for d in dims], torch.float32)
    out = torch.full((int(dims[1]), R), 3.0, device="cuda")
    t.mttkrp(1, Fd, R, out=out, accumulate=True, variant=A.DETERMINISTIC)
    fresh = t.mttkrp(1, Fd, R, variant=A.DETERMINISTIC)
    np.testing.assert_allclose(out.cpu().numpy(), 3.0 + fresh.cpu().numpy(), rtol=1e-6)


def test_deterministic_accumulates_and_rejects_unsupported():
    import torch

    dims = np.array([300, 200, 100], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 30000, seed=16)
    R = 16
    rng = np.random.default_rng(5)
    Fd = to_dev([rng.uniform(-1, 1, (int(d), R)) for d in dims], torch.float32)
    t = A.create_alto(dims, cidx, vals)
    base = torch.ones((200, R), device="cuda")
    out = base.clone()
    t.mttkrp(1, Fd, R, out=out, accumulate=True, variant=A.DETERMINISTIC)
    fresh = t.mttkrp(1, Fd, R, variant=A.DETERMINISTIC)
    np.testing.assert_allclose(out.cpu().numpy(), base.cpu().numpy() + fresh.cpu().numpy(), rtol=1e-6, atol=1e-6)
    Fd10 = to_dev([rng.uniform(-1, 1, (int(d), 10)) for d in dims], torch.float32)
    with pytest.raises(A.AltoError):
        t.mttkrp(0, Fd10, 10, variant=A.DETERMINISTIC)
    with pytest.raises(A.AltoError):
        t.mttkrp(0, [f.to(torch.bfloat16) for f in Fd], R, variant=A.DETERMINISTIC)


# ------------------------------------------------------------ long walks

def check_long(dims, nnz, R, variant, seed):
    """Every mode's MTTKRP of nnz random nonzeros with positive values and
    factors against float64 sums, element by element.  An output element is a
    sum of positive products, so its relative error is at most the number of
    float32 roundings on the way of a product to it: a few products, and fewer
    than 1000 additions (a lane group's run, its meeting with the others', and
    the block's or the atomics' chain), 2^-24 each."""
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    idx = [torch.randint(0, d, (nnz,), generator=g, device="cuda") for d in dims]
    vals = torch.rand(nnz, generator=g, device="cuda") + 0.5
    F = [torch.rand((d, R), generator=g, device="cuda") + 0.5 for d in dims]
    t = A.create_alto(np.array(dims, np.uint64), idx, vals)
    for m in range(len(dims)):
        want = torch.zeros((dims[m], R), dtype=torch.float64, device="cuda")
        for a in range(0, nnz, 1 << 21):
            p = vals[a:a + (1 << 21)].double()[:, None].expand(-1, R)
            for j in range(len(dims)):
                if j != m:
                    p = p * F[j][idx[j][a:a + (1 << 21)]].double()
            want.index_add_(0, idx[m][a:a + (1 << 21)], p)
        got = t.mttkrp(m, F, R, variant=variant).double()
        assert bool(((got - want).abs() <= 1000 * 2.0 ** -24 * want).all()), m


@pytest.mark.parametrize("nnz", [(8 << 20) - 1, 8 << 20, (8 << 20) + 1237])
@pytest.mark.parametrize("dims,R", [([1200000, 40, 1100000], 32), ([3000, 40, 2000], 32), ([4200000, 7, 4300000], 8)])
def test_long_sorted_walks(dims, R, nnz):
    """Around the length from which a walk over input factors larger than L2
    (first and last dims, every mode) has two steps of rows in the air."""
    check_long(dims, nnz, R, A.SORTED, seed=nnz % 97)


@pytest.mark.parametrize("dims,nnz", [([1, 5, 200000], 7100003), ([1, 5, 200000], 14200001),
                                      ([9, 1, 300, 2000, 30000], 7100003)])
def test_deterministic_chunks_of_several_tiles(dims, nnz):
    """The deterministic walk's blocks have one tile each up to 7.08M nonzeros;
    above, a block carries its open run from tile to tile: through all of them (a
    mode of one row), through some (a few rows), and not at all (a long mode)."""
    check_long(dims, nnz, 8, A.DETERMINISTIC, seed=len(dims))


@pytest.mark.parametrize("rows,nnz", [(60, 3000), (500, 50000), (500, 1000000)])
def test_deterministic_error_of_short_runs(rows, nnz):
    """Runs that fill a part of a block meet there from many lane groups.  Rounding
    a float32 result costs 2.53e-8 rms over evenly spread mantissas, and a chain of n
    equal parts sqrt(n / 3) of that: the runs here may cost as much as one of 14."""
    import torch

    R, seeds, sq, dims = 8, 6, 0.0, [rows, 3000, 4000]
    for seed in range(seeds):
        g = torch.Generator(device="cuda").manual_seed(seed)
        cidx = torch.stack([torch.randint(0, d, (nnz,), device="cuda", generator=g) for d in dims])
        vals = torch.rand(nnz, device="cuda", generator=g)
        F = [torch.rand((d, R), device="cuda", generator=g) * torch.exp2(torch.rand(R, device="cuda", generator=g))
             for d in dims]
        t = A.AltoTensor(dims, cidx, vals)
        out = t.mttkrp(0, F, R, variant=A.DETERMINISTIC).double()
        ref = torch.zeros_like(out)
        ref.index_add_(0, cidx[0], vals.double()[:, None] * F[1].double()[cidx[1]] * F[2].double()[cidx[2]])
        sq += float((((out - ref) / ref.clamp(min=1e-30)) ** 2).mean()) / seeds
        t.close()
    assert sq ** 0.5 <= (14 / 3) ** 0.5 * 2.53e-8, sq ** 0.5


@pytest.mark.parametrize("dims,per", [([300, 400, 500], 16), ([30, 40, 50, 60], 20), ([30, 40, 50, 60, 7], 24)])
def test_row_sorted_copy_bytes(dims, per):
    """A decoded copy is its records (and 16 of padding), and nothing else."""
    import torch

    rng = np.random.default_rng(5)
    nnz = 20000
    t = A.create_alto(np.array(dims, np.uint64), np.stack([rng.integers(0, d, nnz) for d in dims]).astype(np.uint64),
                      rng.random(nnz))
    before = t.device_bytes()
    F = [torch.rand((d, 16), device="cuda") for d in dims]
    t.mttkrp(0, F, 16, variant=A.SORTED)
    assert t.device_bytes() - before == (nnz + 16) * per


@pytest.mark.parametrize("dims,nnz,R", [
    ([2730, 5, 30], 3001, 3),  # 32,760 bytes of rows: staged
    ([2731, 5, 30], 3001, 3),  # 32,772: not; 5 rows: a full grid of staging blocks
    ([7, 600, 40, 3, 50, 60], 20003, 1),
    ([70, 300], 4099, 10),
    ([62, 11, 40, 9], 9001, 130),  # two windows of columns, of 128 and 2
    ([1, 3, 2, 2, 2, 2, 2, 2], 40, 5)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_any_rank_line_of_few_rows(dims, nnz, R, dtype):
    import torch

    rng = np.random.default_rng(nnz)
    cidx = np.stack([rng.integers(0, d, nnz) for d in dims]).astype(np.uint64)
    check_modes(dims, cidx, rng.uniform(-1.0, 1.0, nnz), R, (A.ATOMIC, A.AUTO), getattr(torch, dtype))


# ------------------------------------------------------------ shards

@pytest.mark.parametrize("nparts", [1, 3, 8])
def test_shards_sum_to_the_whole(nparts):
    """alto_tensor_restrict: the shards' MTTKRPs add up to the whole
    tensor's, and each shard keeps the exact keys of its line range."""
    import torch

    from alto_b200 import shard

    dims = np.array([4800000, 1800000, 1800000], np.uint64)
    cidx, vals = synth.powerlaw_coo(dims, 100000, [1.2, 1.2, 1.2], seed=21, values="lognormal")
    R = 32
    rng = np.random.default_rng(7)
    Fd = to_dev([rng.uniform(-1, 1, (int(d), R)) for d in dims], torch.float32)
    whole = A.create_alto(dims, cidx, vals)
    keys = whole.export()
    parts = [shard.shard_tensor(A.create_alto(dims, cidx, vals), p, nparts) for p in range(nparts)]
    assert sum(p.nnz for p in parts) == whole.nnz
    off = 0
    for p in parts:
        k = p.export()
        assert np.array_equal(k["idx"], keys["idx"][off:off + p.nnz])
        off += p.nnz
    for m in range(3):
        ref = whole.mttkrp(m, Fd, R).cpu().numpy()
        tot = sum(p.mttkrp(m, Fd, R, variant=v).cpu().numpy() for p in parts for v in (A.AUTO,))
        assert rel_err(tot, ref) <= 1e-5


def test_freeing_a_tensor_leaves_another_threads_capture():
    """Destroying a handle waits for the device; a capture that another thread
    has under way (not in global mode) goes on."""
    import threading

    import torch

    dims = np.array([50, 60, 70], np.uint64)
    cidx, vals = synth.uniform_coo(dims, 5000, seed=1)
    t = A.create_alto(dims, cidx, vals)
    x = torch.zeros(1000, device="cuda")
    x.add_(1.0)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        x.add_(1.0)
        held = [t]
        del t
        th = threading.Thread(target=held.clear)
        th.start()
        th.join()
        x.add_(1.0)
    g.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 3000.0


def long_tensor(seed):
    """A tensor of 2M nonzeros and factors, the inputs of the tests below."""
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dims = [3000, 2000, 1000]
    idx = [torch.randint(0, d, (2000000,), generator=g, device="cuda") for d in dims]
    vals = torch.rand(2000000, generator=g, device="cuda")
    F = [torch.rand((d, 16), generator=g, device="cuda") for d in dims]
    return np.array(dims, np.uint64), idx, vals, F


def test_freeing_a_tensor_waits_for_work_on_other_streams():
    """A tensor destroyed while another stream still walks it: the walks end
    first, and what is then made in its memory does not reach them."""
    import torch

    dims, idx, vals, F = long_tensor(3)
    _, other, vals2, _ = long_tensor(4)
    side, third = torch.cuda.Stream(), torch.cuda.Stream()
    results, ended = [], []
    for early in (False, True):
        t = A.create_alto(dims, idx, vals)
        out = torch.zeros((int(dims[0]), 16), device="cuda")
        t.mttkrp(0, F, 16, out=out, variant=A.DETERMINISTIC)  # (builds the row-sorted copy)
        done = torch.cuda.Event()
        torch.cuda.synchronize()
        for _ in range(1500):  # about 0.1 s of device time, 0.02 s to queue
            t.mttkrp(0, F, 16, out=out, accumulate=True, variant=A.DETERMINISTIC, stream=side)
        done.record(side)
        if not early:
            torch.cuda.synchronize()
        t.close()
        ended.append(done.query())
        u = A.create_alto(dims, other, vals2, stream=third)  # same sizes, other contents
        torch.cuda.synchronize()
        results.append(out)
        u.close()
    assert all(ended)
    assert torch.equal(*results)


def test_first_use_inside_a_capture_is_refused():
    """A call that has to allocate is refused under a stream capture (the copy it
    would build there would only be captured, not made), and works after it."""
    import torch

    rt = pytest.importorskip("cuda.bindings.runtime")
    dims, idx, vals, F = long_tensor(5)
    t = A.create_alto(dims, idx, vals)
    out = torch.zeros((int(dims[1]), 16), device="cuda")
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    for mode in (rt.cudaStreamCaptureMode.cudaStreamCaptureModeGlobal,
                 rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal):
        rt.cudaStreamBeginCapture(s.cuda_stream, mode)
        try:
            with pytest.raises(A.AltoError):
                t.mttkrp(1, F, 16, out=out, variant=A.SORTED, stream=s)
        finally:
            err, graph = rt.cudaStreamEndCapture(s.cuda_stream)
        assert err != rt.cudaError_t.cudaSuccess
        rt.cudaGetLastError()
    t.mttkrp(1, F, 16, out=out, variant=A.SORTED, stream=s)
    s.synchronize()
    want = A.create_alto(dims, idx, vals).mttkrp(1, F, 16, variant=A.ATOMIC)
    assert float((out - want).abs().max() / want.abs().max()) <= TOL
