"""Launches take the autotuner's choices, for whole transforms and for the strided
passes of large ones."""
import numpy as np
import pytest

import benchntt_b200 as bn
import common as C

pytestmark = pytest.mark.gpu

Q_GENERAL = 0xB504F333F9DE6484597D89B3754ABE9


@pytest.fixture(scope="module")
def ctx():
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    c = bn.Context(0, stream=stream.cuda_stream)
    c.torch_stream = stream
    yield c
    bn.lib().bntt_autotune_reset()
    c.close()


@pytest.fixture
def force(ctx, tmp_path):
    """Installs exactly the given choices, as a file of the tuner."""
    full = tmp_path / "full.tune"
    ctx.autotune(str(full))
    head = full.read_text().splitlines()[0]

    def install(*lines):
        f = tmp_path / "forced.tune"
        f.write_text("\n".join([head, *lines]) + "\n")
        bn.lib().bntt_autotune_reset()
        ctx.autotune_load(str(f))

    yield install
    bn.lib().bntt_autotune_reset()


def microseconds(ctx, plan, logn, batch):
    """of one forward launch sequence, from a captured graph"""
    import torch
    x = torch.from_numpy(np.resize(C.uniform_pairs(3, 1 << logn, plan.q), (batch << logn, 2)).view(np.int64)).cuda()
    y = torch.empty_like(x)
    plan.forward(y, x, batch)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=ctx.torch_stream):
        for _ in range(10):
            plan.forward(y, x, batch)
    best = float("inf")
    with torch.cuda.stream(ctx.torch_stream):
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 100)
    return best


def plan_of(ctx, logn, q):
    return bn.Plan(ctx, logn, q, (1 << 251) // q, C.uniform_pairs(4 + logn, 1 << logn, q))


def pair(ctx, force, logn, q, batch, *lines):
    """(untuned, tuned) time of a launch"""
    bn.lib().bntt_autotune_reset()
    plain = plan_of(ctx, logn, q)
    force(*lines)
    tuned = plan_of(ctx, logn, q)
    times = microseconds(ctx, plain, logn, batch), microseconds(ctx, tuned, logn, batch)
    plain.close()
    tuned.close()
    return times


# 16 elements per thread and one resident CTA with the general multiply: slower than
# the default by more than a tenth, which shows that the choice is taken
def test_large_launches_take_the_strided_choice(ctx, force):
    plain, tuned = pair(ctx, force, 16, Q_GENERAL, 64, "sub 6 1 0 4 8 1 0")
    assert tuned > 1.1 * plain, (plain, tuned)


SHAPES = ([(m, 1, 4, 8, 1) for m in (5, 6, 7)] + [(m, 1, 2, 1024 >> m, 4) for m in (5, 6, 7)] +
          [(m, 0, 4, 8, 1) for m in (5, 6, 7)] + [(m, 0, 2, 1024 >> m, 4) for m in (5, 6, 7)])


# 2^13 = 5 + 8, 2^16 = 6 + 10 and 2^17 = 7 + 10 stages: the strided choice, and for
# the last pass a staged shape (not one that copies the table, which whole
# transforms take); more than 2^20 elements, in a ragged number of transforms
@pytest.mark.parametrize("m,fast,logr,tpc,minb", SHAPES, ids=lambda v: str(v))
def test_strided_choices_match_oracle(ctx, force, m, fast, logr, tpc, minb):
    import torch
    logn, last = {5: (13, 8), 6: (16, 10), 7: (17, 10)}[m]
    q = C.Q_NTT if fast else Q_GENERAL
    mu = (1 << 251) // q
    lines = [f"sub {m} 1 {fast} {logr} {tpc} {minb} 0"]
    if fast:
        lines.append(f"sub {last} 0 1 2 {1024 >> last} 4 {1 if m == 6 else 3}")
    force(*lines)
    n, rows, batch = 1 << logn, 2, (1 << 20 >> logn) + 3
    x, t = C.uniform_pairs(8 + m, rows * n, q), C.uniform_pairs(4 + logn, n, q)
    plan = bn.Plan(ctx, logn, q, mu, t)
    at = ((np.arange(batch) % rows)[:, None] * n + np.arange(n)).reshape(-1)
    dx = torch.from_numpy(x[at].view(np.int64)).cuda()
    dy = torch.empty_like(dx)
    plan.forward(dy, dx, batch)
    torch.cuda.synchronize()
    want = C.oracle_ntt(x, t, logn, q, mu, form=1, threads=8)
    assert np.array_equal(dy.cpu().numpy().view(np.uint64), want[at])
    plan.close()


def test_files_of_earlier_versions_load(ctx, force):
    """Strided passes of 8 to 10 stages are no longer timed; files that name their
    shapes load as before, and shapes that never were are refused as before."""
    force("sub 8 1 0 4 8 1 0", "sub 9 1 0 4 4 1 0", "sub 10 1 0 4 4 1 0", "sub 8 1 1 4 8 1 0", "sub 9 1 1 4 4 3 0",
          "sub 9 1 1 4 8 1 0", "sub 10 1 1 4 8 1 0", "sub 10 1 1 4 4 1", "sub 10 0 1 2 1 4 0", "sub 7 1 1 2 8 4 0")
    for line in ("sub 9 1 0 4 8 1 0", "sub 9 1 1 4 2 1 0", "sub 8 1 1 3 8 1 0", "sub 10 1 1 4 4 3 0", "sub 8 1 1 4 8 1 1"):
        with pytest.raises(bn.BnttError) as e:
            force(line)
        assert e.value.status == bn.EINVAL
