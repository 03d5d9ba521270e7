"""Which launches take the autotuner's choices: those that are not much smaller
than the launches it times, for whole transforms and for the strided passes of
large ones.  A small launch keeps its own default.
"""
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


# The same kernel in both cases, or one that the tuner would not choose here: one
# transform of 2^8 with the shape of large launches takes 1.6 times as long.
@pytest.mark.parametrize("logn,line", [(8, "sub 8 0 1 3 2 10 0"), (10, "sub 10 0 1 3 1 7 0"), (9, "sub 9 0 1 3 4 3 0")])
def test_one_transform_keeps_its_shape(ctx, force, logn, line):
    plain, tuned = pair(ctx, force, logn, C.Q_NTT, 1, line)
    assert tuned < 1.2 * plain, (plain, tuned)


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


@pytest.mark.parametrize("src", [1, 3])
@pytest.mark.parametrize("layout", [bn.LAYOUT_HILO, bn.LAYOUT_U128])
def test_staged_kernels_with_a_fused_product(ctx, force, src, layout):
    """The staged kernels in a launch that takes them, with the pointwise product of
    the last pass, in both layouts."""
    import torch
    force(f"sub 7 0 1 2 8 4 {src}")
    logn, n, rows, batch = 7, 128, 3, (1 << 13) + 3
    order = (lambda a: a) if layout == bn.LAYOUT_HILO else (lambda a: np.ascontiguousarray(a[:, ::-1]))
    x, b, t = (C.uniform_pairs(seed, count, C.Q_NTT) for seed, count in ((51, rows * n), (52, rows * n), (53, n)))
    at = ((np.arange(batch) % rows)[:, None] * n + np.arange(n)).reshape(-1)
    plan = bn.Plan(ctx, logn, C.Q_NTT, C.MU_NTT, order(t), layout)
    dx, db = (torch.from_numpy(order(a)[at].view(np.int64)).cuda() for a in (x, b))
    dy = torch.empty_like(dx)
    plan.forward_mul(dy, dx, db, True, batch)
    torch.cuda.synchronize()
    want = C.oracle_blas("vvmul", C.oracle_ntt(x, t, logn, threads=8), b, C.Q_NTT, C.MU_NTT)
    assert np.array_equal(dy.cpu().numpy().view(np.uint64), order(want)[at])
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
