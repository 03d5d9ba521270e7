"""Job lists that do not fill the device: the persistent kernel takes them with
more threads per tile, and hands every tile to a CTA of its own.  Lists on both
sides of that choice against the oracle, and short lists against the time of the
plan kernels on the same transforms.
"""
import numpy as np
import pytest

import benchntt_b200 as bn
import common as C

pytestmark = pytest.mark.gpu

Q_NC = C.from_pairs(np.load(f"{C.GOLDEN}/ref_gen.npz")["nc_q"])[0]
Q_GENERAL = 0xB504F333F9DE6484597D89B3754ABE9
MU = {q: (1 << 251) // q for q in (Q_NC, Q_GENERAL)}


@pytest.fixture(scope="module")
def ctx():
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    c = bn.Context(0, stream=stream.cuda_stream)
    c.torch_stream = stream
    yield c
    c.close()


class Jobs:
    """A job list over one buffer, with its engine."""

    def __init__(self, ctx, logns, q, layout=bn.LAYOUT_HILO):
        import torch
        self.logns, self.sizes = logns, sorted(set(logns))
        self.order = (lambda a: a) if layout == bn.LAYOUT_HILO else (lambda a: np.ascontiguousarray(a[:, ::-1]))
        self.tables = {n: C.uniform_pairs(50 + n, 1 << n, q) for n in self.sizes}
        self.plans = [bn.Plan(ctx, n, q, MU[q], self.order(self.tables[n]), layout) for n in self.sizes]
        self.offs = np.cumsum([0] + [1 << n for n in logns])
        # few distinct transforms, so that the oracle computes only those
        rows = {n: C.uniform_pairs(60 + n, 3 << n, q).reshape(3, 1 << n, 2) for n in self.sizes}
        self.rows, self.which = rows, [i % 3 for i in range(len(logns))]
        x = np.concatenate([rows[n][k] for n, k in zip(logns, self.which)])
        self.x = torch.from_numpy(self.order(x).view(np.int64)).cuda()
        self.y = torch.empty_like(self.x)
        self.engine = bn.Batch(ctx, self.plans)
        at = (16 * self.offs[:-1]).tolist()
        self.jobs = bn.Batch.jobs([self.x.data_ptr() + o for o in at], [self.y.data_ptr() + o for o in at],
                                  [self.sizes.index(n) for n in logns])

    def results(self):
        import torch
        torch.cuda.synchronize()
        assert self.engine.status() == bn.OK
        return self.order(self.y.cpu().numpy().view(np.uint64))

    def want(self, one):
        """one(rows, table, log2n) for every job"""
        done = {(n, k): one(self.rows[n][k], self.tables[n], n) for n in self.sizes for k in range(3)}
        return np.concatenate([done[n, k] for n, k in zip(self.logns, self.which)])

    def __enter__(self):
        return self

    def __exit__(self, *_):
        self.engine.close()
        for p in self.plans:
            p.close()


# items in one wave of the long lists' kernel: 7 CTAs on each of the SMs
def lists(sms):
    wave = 7 * sms
    mixed = [n for n in range(1, 12) for _ in range(5)] + [13, 16]
    return {"one": [10], "mixed": mixed, "ragged": [4] * 65 + [1] * 257 + [9] * 3,
            "wave": [10] * wave, "wave+1": [10] * (wave + 1), "long": mixed + [9] * (2 * wave), "large": [17, 20]}


@pytest.mark.parametrize("name", ["one", "mixed", "ragged", "wave", "wave+1", "long", "large"])
@pytest.mark.parametrize("q,layout", [(Q_NC, bn.LAYOUT_HILO), (Q_NC, bn.LAYOUT_U128), (Q_GENERAL, bn.LAYOUT_HILO)],
                         ids=["hilo", "u128", "general"])
def test_lists_match_oracle(ctx, name, q, layout):
    with Jobs(ctx, lists(ctx.sm_count)[name], q, layout) as j:
        j.engine.run_dev(j.jobs)
        assert np.array_equal(j.results(), j.want(lambda x, t, n: C.oracle_ntt(x, t, n, q, MU[q], form=1, threads=8)))
        if q == Q_NC:
            j.y.zero_()
            j.engine.run_inverse_dev(j.jobs)
            assert np.array_equal(j.results(), j.want(lambda x, t, n: C.oracle_ntt_inverse(x, t, n, q, MU[q])))


# A tile of a list costs what it costs a plan's launch, plus its item (a few
# loads) and the list's launch (a memset before the kernel, about 5 us): 1.2 to
# 1.3 times the plan's time here.  A list whose CTAs run two tiles in a row while
# others have none takes twice the time.
LIMIT = 1.6


def fastest(ctx, call, reps):
    """us of one call, the fastest of ten runs of `reps`"""
    import torch
    best = float("inf")
    with torch.cuda.stream(ctx.torch_stream):
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(reps):
                call()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3 / reps)
    return best


@pytest.mark.parametrize("q,inverse", [(Q_NC, False), (Q_NC, True), (Q_GENERAL, False)],
                         ids=["forward", "inverse", "general"])
@pytest.mark.parametrize("logn,count", [(10, 592), (10, 1036), (20, 1)])
def test_short_lists_take_about_a_plans_time(ctx, q, inverse, logn, count):
    import torch
    with Jobs(ctx, [logn] * count, q) as j:
        plan = j.plans[0]
        call = (lambda: plan.inverse(j.y, j.x, count)) if inverse else (lambda: plan.forward(j.y, j.x, count))
        call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()   # so that the host does not set the pace of the plan's calls
        with torch.cuda.graph(graph, stream=ctx.torch_stream):
            for _ in range(20):
                call()
        alone = fastest(ctx, graph.replay, 2) / 20
        listed = fastest(ctx, lambda: (j.engine.run_inverse_dev if inverse else j.engine.run_dev)(j.jobs), 40)
        assert listed < LIMIT * alone, (listed, alone)
