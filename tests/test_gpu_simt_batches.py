"""FP32 forward batches and chunk sizes: a field beside a wider one keeps its own spot chunks, so it gives
the same bits as alone and takes the same time; a lattice of more than 60 spots still runs two blocks to
an SM.  Times are device times, the least of several, in turn; each bound lies between the two times
measured (given at the test)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pb():
    return importlib.import_module("gpu-proton-dose-engine_b200")


def _problem(pb, nx, ny, nz, nsx, nsy, nl, seed=0):
    rng = np.random.default_rng(seed)
    grid = pb.model.DoseGrid(nx, ny, nz, 0.2, 0.2, 0.2, -0.1 * nx, -0.1 * ny, 0.0)
    lat = pb.model.SpotLattice(nsx, nsy, nl, 0.25, 0.25, 0.03, -0.02, weights=rng.uniform(0.1, 1.0, (nl, nsy, nsx)))
    return pb.model.PBProblem(grid, lat, rng.uniform(0.5, 2.0, (nl, nz)), rng.uniform(0.25, 0.8, (nl, nz)))


def _batch(pb, probs):
    import torch
    lib = pb._lib
    jobs, keep, doses = (lib.Job * len(probs))(), [], []
    for k, p in enumerate(probs):
        w = torch.as_tensor(np.float32(p.lattice.weights), device="cuda")
        i, s = (torch.as_tensor(a, device="cuda") for a in (p.idd, p.sigma))
        d = torch.empty(p.grid.shape, dtype=torch.float32, device="cuda")
        jobs[k] = lib.Job(field=lib.field_of(p), w=lib.ptr(w), idd=lib.ptr(i), sigma=lib.ptr(s), dose=lib.ptr(d))
        keep += [w, i, s]
        doses.append(d)
    prec = lib.PREC["fp32"]
    ws = torch.empty(lib.query("pbd_forward_batch_workspace", jobs, len(probs), prec), dtype=torch.uint8,
                     device="cuda")

    def run(_keep=keep):
        lib.call("pbd_forward_batch", jobs, len(probs), prec, lib.ptr(ws), ws.numel(), lib.stream_handle())
        return doses

    return run


def _times(*calls, reps=10, rounds=6):
    import torch
    best = [float("inf")] * len(calls)
    for _ in range(rounds):
        for k, f in enumerate(calls):
            f()
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(reps):
                f()
            b.record()
            b.synchronize()
            best[k] = min(best[k], a.elapsed_time(b) / reps)
    return best


@pytest.mark.parametrize("lattices", [((41, 41), (73, 73)), ((65, 9), (64, 64), (1, 129)), ((49, 70), (3, 48))])
def test_batch_gives_each_job_its_bits(pb, lattices):
    import torch
    probs = [_problem(pb, 90 + 13 * k, 60 + 31 * k, 3, nsx, nsy, 2, seed=k) for k, (nsx, nsy) in enumerate(lattices)]
    got = [d.clone() for d in _batch(pb, probs)()]
    for p, d in zip(probs, got):
        assert torch.equal(d, _batch(pb, [p])()[0])


def test_wide_job_leaves_the_others_their_chunks(pb):
    """Three 41 x 41 fields with and without a small one of 73 x 73 spots."""
    a = [_problem(pb, 128, 128, 64, 41, 41, 12, seed=k) for k in range(3)]
    alone, both = _times(_batch(pb, a), _batch(pb, a + [_problem(pb, 64, 64, 8, 73, 73, 2)]))
    assert both <= 1.14 * alone          # 1.27 times with one chunk size for the batch, 1.01 with its own


def test_uneven_lattice_has_a_chunk_per_axis(pb):
    """41 spots beside 73 of the other axis take about as long as 40."""
    p40, p41 = (_problem(pb, 128, 128, 64, 73, n, 10) for n in (40, 41))
    t40, t41 = _times(_batch(pb, [p40]), _batch(pb, [p41]))
    assert t41 <= 1.2 * t40              # 1.39 times with one chunk size for both axes, 1.02 with one each


def test_more_than_60_spots_run_two_blocks_to_an_sm(pb):
    """Chunks of 64 spots take the most shared memory: 61 spots take about as long as 60."""
    p60, p61 = (_problem(pb, 200, 200, 64, n, n, 10) for n in (60, 61))
    t60, t61 = _times(_batch(pb, [p60]), _batch(pb, [p61]))
    assert t61 <= 1.12 * t60             # 1.26 times with one block to an SM, 1.01 with two
