"""The wavefront schedule's own paths: RANMAR as a warp produces it, phantoms
whose axes end after one or a few voxels (the photon flight's last planes,
the boundary steps' region changes, vacuum voxels inside), and history counts
around a warp and a block of queue records."""

import numpy as np
import pytest
from cases import run_seeds
from stats import compare, consistent

from ompmc_gb300 import api, data
from ompmc_gb300 import workloads as W


def _warp_ranmar(u, steps):
    """`steps` x 32 numbers of the stream with seed words u[1..97], the way
    RngPool::refill does it: word q is the value of lane `lane` `age` steps
    ago, lane l starts from Weyl term 362436 - (l + 1) * 7654321 + one step."""
    mod, inc = 16777213, 7654321
    lanes = np.arange(32)
    v = np.zeros((5, 32), np.int64)  # v[a]: the lanes' values a steps ago
    for q in range(1, 98):
        age = (q - 1) // 32 + 1 if q <= 96 else 4
        v[age, 32 * age - q if q <= 96 else 31] = u[q - 1]
    c = (362436 - (lanes + 1) * inc + 32 * inc) % mod
    out = []
    for _ in range(steps):
        x33 = np.roll(np.where(lanes == 31, v[2], v[1]), 1)
        x97 = np.roll(np.where(lanes == 31, v[4], v[3]), 1)
        v[2:] = v[1:-1].copy()
        v[1] = (x97 - x33) & 0xFFFFFF
        c = (c - 32 * inc) % mod
        out.append((v[1] - c) & 0xFFFFFF)
    return np.concatenate(out)


def _seed_words(ixx, jxx):
    """initRandom's 97 words (omc_random.c:97-114)."""
    i, j, k, m = ixx // 177 % 177 + 2, ixx % 177 + 2, jxx // 169 % 178 + 1, jxx % 169
    u = []
    for _ in range(97):
        s, t = 0, 8388608
        for _ in range(24):
            n = i * j % 179 * k % 179
            i, j, k = j, k, n
            m = (53 * m + 1) % 169
            if m * n % 64 >= 32:
                s += t
            t //= 2
        u.append(s)
    return u


@pytest.mark.parametrize("seeds", [(97, 33), (1802, 9373), (31328, 1)])
def test_warp_form_of_ranmar_is_the_stream(seeds, oracle):
    np.testing.assert_array_equal(_warp_ranmar(_seed_words(*seeds), 20), oracle.ranmar(*seeds, 640))


def test_turned_numbers_of_a_recurrence_fall_on_three_lanes():
    """x[n], x[n-33] and x[n-97] end on lanes l - r(s), l - 1 - r(s-1) and
    l - 1 - r(s-3), r turning by 5 a step (kPoolTurn)."""
    for s in range(32):
        r = [5 * (s - d) % 32 for d in range(4)]
        lanes = {-r[0] % 32, (-1 - r[1]) % 32, (-1 - r[3]) % 32}
        assert len(lanes) == 3


def _problem(tmp_path, shape, charge, energy, vacuum, histories, nbatch):
    """A box of uneven voxels, water and lung slabs, one vacuum layer when
    asked for."""
    nx, ny, nz = shape
    rng = np.random.default_rng(nx * 100 + ny * 10 + nz)
    edges = [np.concatenate(([0.0], np.cumsum(rng.uniform(0.4, 1.6, n)))) for n in shape]
    xb, yb, zb = (10.0 / e[-1] * e - (5.0 if k < 2 else 0.0) for k, e in enumerate(edges))
    med = np.ones((nz, ny, nx), np.uint8)
    rho = np.ones((nz, ny, nx))
    med[nz // 2:], rho[nz // 2:] = 2, 0.26
    if vacuum and nz > 2:
        med[1], rho[1] = 0, 0.0
    P = data.paths()
    job = W.Job("(in memory)", P["pegs"], P["pgs4form"], P["data_folder"], str(tmp_path) + "/", mono_energy=energy,
                charge=charge, ncase=histories, nbatch=nbatch, collimator=(-3.0, 3.0, -3.0, 3.0), ssd=60.0)
    return api.Problem(api.Input(text=job.text()), phantom=api.Phantom.from_arrays([W.WATER, W.LUNG], xb, yb, zb, med,
                                                                                  rho))


@pytest.mark.gpu
@pytest.mark.parametrize("shape,charge,energy,vacuum", [((1, 1, 1), 0, 3.0, False), ((1, 7, 2), 0, 3.0, False),
                                                        ((33, 1, 5), 0, 0.2, True), ((2, 3, 17), 0, 6.0, True),
                                                        ((3, 1, 9), -1, 5.0, True), ((1, 4, 6), 1, 5.0, False)])
@pytest.mark.parametrize("precision", [api.FP32, api.FP64])
def test_edges_of_the_phantom(shape, charge, energy, vacuum, precision, tmp_path, engine, oracle):
    """Per-voxel dose and total energy against the oracle (charged particles
    with vacuum voxels: against the per-lane schedule): consistent at p > 1e-4
    where there are voxels enough, the total within 5 sigma of the two runs'
    batch totals."""
    nb, n = 20, 20 * (10000 if charge == 0 else 2000)
    prob = _problem(tmp_path, shape, charge, energy, vacuum, n, nb)
    engine.load(prob)
    a, a2, st = engine.run(precision=precision, seeds=run_seeds(3))
    assert st.error_flags == 0 and st.histories == n
    totals = engine.batch_sums(np.concatenate(([0.0], np.ones(prob.nreg - 1))))
    if charge and vacuum:
        ref, ref2, _ = engine.run(precision=precision, seeds=run_seeds(4), schedule=api.LANES)
    else:
        ref, ref2, _ = oracle.run(prob, seeds=run_seeds(4), nthreads=0)
    sigma = np.sqrt(2.0 * nb) * totals.std(ddof=1)
    assert abs(a[1:].sum() - ref[1:].sum()) < 5.0 * sigma, (a[1:].sum(), ref[1:].sum(), sigma)
    c = compare(a, a2, ref, ref2, nb)
    if c["n"] >= 10:
        assert consistent(c), c


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [api.FP32, api.FP64])
@pytest.mark.parametrize("history_stats", [0, 1])
@pytest.mark.parametrize("nperbatch", [1, 31, 32, 33, 1023])
def test_few_histories(nperbatch, history_stats, precision, tmp_path, engine):
    """Chunks of one to 32 particles: every history is transported once, no
    energy appears (photons that leave are not scored), and history scoring
    merges every history once, also where warps have lanes without a
    particle."""
    prob = _problem(tmp_path, (5, 4, 6), -1, 5.0, False, 2 * nperbatch, 2)
    engine.load(prob)
    a, _, st = engine.run(precision=precision, history_stats=history_stats)
    assert st.error_flags == 0 and st.histories == 2 * nperbatch
    assert abs(st.ensrc - 5.0 * 2 * nperbatch) < 1e-6 * st.ensrc
    assert 0.0 < a.sum() < (1.0 + 1e-4) * st.ensrc  # 1e-4: FP32 energy losses over some hundred steps
    if history_stats:
        s, _, merged, split = engine.history_sums()
        assert merged == 2 * nperbatch and split == 0
        np.testing.assert_allclose(s, a, rtol=1e-9, atol=1e-12 * a.max())


@pytest.mark.gpu
def test_continued_streams_of_the_two_schedules_do_not_repeat(tmp_path, engine):
    """A run that continues the streams draws new numbers, whichever schedule
    ran before."""
    prob = _problem(tmp_path, (4, 4, 4), 0, 3.0, False, 20000, 2)
    engine.load(prob)
    runs = []
    for schedule in (api.WAVEFRONT, api.WAVEFRONT, api.LANES, api.WAVEFRONT):
        _, _, st = engine.run(precision=api.FP32, schedule=schedule, nlanes=0, continue_streams=1 if runs else 0)
        assert st.error_flags == 0
        runs.append(st.deposits)
    assert len(set(runs)) == len(runs)
