"""Launches that overlap the kernel before them in the stream must still see all
of its writes and leave its inputs alone: dependent chains of plan and vector
calls on shared buffers, with foreign kernels and copies in between, run
directly and from a captured graph with a fork to a second stream.  Compared bit
for bit with the oracle's steps one after the other.
"""
import functools

import numpy as np
import pytest

import benchntt_b200 as bn
import common as C

pytestmark = pytest.mark.gpu

GEN = np.load(f"{C.GOLDEN}/ref_gen.npz")
Q = C.from_pairs(GEN["nc_q"])[0]
MU = (1 << 251) // Q
ROOT21 = C.from_pairs(GEN["nc_root21"])[0]


@functools.cache
def table(logn):
    return C.negacyclic_table(Q, logn, pow(ROOT21, 1 << (C.NC_LOG2_ORDER - logn - 1), Q))


def expected(logn, x, b, rounds):
    """`rounds` of y = inverse(forward(x) o b), and forward(x) of the last one"""
    t = table(logn)
    for _ in range(rounds):
        f = C.oracle_ntt(x, t, logn, Q, MU, form=1, threads=8)
        x = C.oracle_ntt_inverse(C.oracle_blas("vvmul", f, b, Q, MU), t, logn, Q, MU)
    return x, f


# lone, few and many elements; one and two passes over memory
@pytest.mark.parametrize("logn,batch", [(4, 1), (10, 3), (7, 2048), (13, 2), (13, 40), (16, 40)])
@pytest.mark.parametrize("graph", [False, True])
def test_dependent_chain(logn, batch, graph):
    torch = pytest.importorskip("torch")
    n, rounds = batch << logn, 2
    x, b = C.uniform_pairs(41 + logn, n, Q), C.uniform_pairs(42 + logn, n, Q)
    want, want_f = expected(logn, x, b, rounds)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()

    s, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    ctx, ctx2 = bn.Context(0, stream=s.cuda_stream), bn.Context(0, stream=s2.cuda_stream)
    plan = bn.Plan(ctx, logn, Q, MU, table(logn))
    x0, db = dev(x), dev(b)
    u, f, side = (torch.zeros_like(x0) for _ in range(3))
    torch.cuda.synchronize()
    plan.inverse(u, u, batch)    # builds the inverse table, outside the capture
    torch.cuda.synchronize()

    def chain():
        u.copy_(x0)
        for _ in range(rounds):
            plan.forward(f, u, batch)
            u.fill_(-1)          # a foreign kernel right after the last read of u
            s2.wait_stream(s)
            bn.blas(ctx, "vvmul", u, f, db, Q, MU)
            with torch.cuda.stream(s2):
                side.copy_(f)    # a second reader of f, on the other stream
                bn.blas(ctx2, "vvadd", side, side, side, Q, MU)
            s.wait_stream(s2)    # f is overwritten by the next round
            plan.inverse(u, u, batch)

    reps = 3
    if graph:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            chain()
        for _ in range(reps):
            u.zero_()
            g.replay()
    else:
        with torch.cuda.stream(s):
            for _ in range(reps):
                chain()
    torch.cuda.synchronize()

    def host(d):
        return d.cpu().numpy().view(np.uint64).reshape(-1, 2)

    assert np.array_equal(host(u), want)
    assert np.array_equal(host(f), want_f)
    assert np.array_equal(host(side), C.oracle_blas("vvadd", want_f, want_f, Q, MU))
    for o in (plan, ctx, ctx2):
        o.close()
