"""Forward transforms on values that leave the common path of the partly
reduced butterflies: sums of exactly q, sums whose low 64 bits equal q's (where
the reference's addmod128 is 2^64 short, src/ntt_scalar.c:49-79), zeros, and
values next to 0 and q, in the inputs and, through tables of 0, 1 and q - 1, in
every later stage.  Compared bit for bit with the oracle.
"""
import numpy as np
import pytest

import benchntt_b200 as bn
import common as C
from gpu_util import DevBuf

Q_NC = C.from_pairs(np.load(f"{C.GOLDEN}/ref_gen.npz")["nc_q"])[0]
MODULI = {"ntt": C.Q_NTT, "blas": C.Q_BLAS, "friendly": Q_NC}   # k = 719, 59 and 0x7bfffff


def pick(rng, values, n):
    return C.to_pairs(values)[rng.integers(0, len(values), size=n)]


def values(kind: str, q: int, logn: int, batch: int):
    """(inputs, table) of `batch` transforms of 2^logn points."""
    rng = np.random.default_rng(1000 * logn + batch)
    n = 1 << logn
    edge = C.edge_values(q)
    if kind == "edges":        # sums of special values in every stage
        return pick(rng, edge, n * batch), pick(rng, [1, q - 1, 0, 1, q - 1], n)
    if kind == "units":        # sums of exactly q
        return pick(rng, [0, 1, q - 1, q], n * batch), pick(rng, [1, q - 1], n)
    if kind == "sparse":       # special values among spread ones
        x, t = C.uniform_pairs(3 + logn, n * batch, q), C.uniform_pairs(4 + logn, n, q)
        at, bt = rng.random(n * batch) < 0.2, rng.random(n) < 0.6
        x[at], t[bt] = pick(rng, edge, int(at.sum())), pick(rng, [1, q - 1], int(bt.sum()))
        return x, t
    # ternary coefficients over a spread table, and transforms of zeros
    x = pick(rng, [0, 1, q - 1], n * batch)
    x[:n] = 0
    return x, C.uniform_pairs(4 + logn, n, q)


def mu_of(q):
    return (1 << 251) // q


def exact_network(x, t, logn, q):
    """The network with exact arithmetic mod q."""
    n = 1 << logn
    v = np.array(C.from_pairs(x), dtype=object)
    tw = np.array(C.from_pairs(t), dtype=object)
    for s in range(logn):
        v = v.reshape(-1, 1 << s, 2, n >> (s + 1))
        p = v[:, :, 1] * tw[1 << s:2 << s].reshape(1, -1, 1) % q
        v = np.stack(((v[:, :, 0] + p) % q, (v[:, :, 0] - p) % q), axis=2)
    return v.reshape(-1)


@pytest.mark.parametrize("q", MODULI.values(), ids=MODULI.keys())
def test_the_values_reach_the_reference_corners(q):
    """Without the reference's two addmod corners the outputs would differ."""
    for kind in ("edges", "units"):
        x, t = values(kind, q, 8, 8)
        y = np.array(C.from_pairs(C.oracle_ntt(x, t, 8, q, mu_of(q))), dtype=object)
        e = exact_network(x, t, 8, q)
        if kind == "units":
            assert (y == q).sum() > 10 and (y[e == 0] == 0).sum() > 10   # q and 0 both occur
        else:
            assert (y % q != e).sum() > 10


@pytest.fixture(scope="module")
def ctx():
    c = bn.Context(0)
    yield c
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["edges", "units", "sparse", "ternary"])
@pytest.mark.parametrize("logn,batch,qn", [(1, 300, "ntt"), (2, 300, "friendly"), (3, 131, "ntt"), (4, 67, "friendly"),
                                           (5, 33, "blas"), (6, 17, "ntt"), (7, 9, "friendly"), (8, 5, "ntt"),
                                           (9, 3, "blas"), (10, 3, "friendly"), (11, 2, "ntt"), (13, 2, "friendly"),
                                           (16, 1, "ntt"), (18, 1, "friendly")])
def test_plan_matches_oracle(ctx, kind, logn, batch, qn):
    q = MODULI[qn]
    x, t = values(kind, q, logn, batch)
    plan = bn.Plan(ctx, logn, q, mu_of(q), t)
    dx, dy = DevBuf.from_array(ctx, x), DevBuf(ctx, x.nbytes)
    bn.check(bn.lib().bntt_ntt_forward_dev(plan.handle, dy.ptr, dx.ptr, batch))
    want = C.oracle_ntt(x, t, logn, q, mu_of(q), form=1, threads=8)
    assert np.array_equal(dy.to_array(), want)
    # fused with a product, in place
    b = C.uniform_pairs(9, x.shape[0], q)
    db = DevBuf.from_array(ctx, b)
    bn.check(bn.lib().bntt_ntt_forward_mul_dev(plan.handle, dx.ptr, dx.ptr, db.ptr, 1, batch))
    assert np.array_equal(dx.to_array(), C.oracle_blas("vvmul", want, b, q, mu_of(q)))
    for d in (dx, dy, db):
        d.free()
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["edges", "units", "sparse", "ternary"])
@pytest.mark.parametrize("layout", [bn.LAYOUT_HILO, bn.LAYOUT_U128])
def test_batch_matches_oracle(ctx, kind, layout):
    """Every size of the persistent kernel, with large jobs of two and three passes."""
    q = Q_NC
    logns = [n for n in range(1, 13) for _ in range(9)] + [15, 16, 18]
    parts = [values(kind, q, n, 1) for n in logns]
    tables = {n: t for n, (_, t) in zip(logns, parts)}
    order = (lambda a: a) if layout == bn.LAYOUT_HILO else (lambda a: np.ascontiguousarray(a[:, ::-1]))
    sizes = sorted(tables)
    plans = [bn.Plan(ctx, n, q, mu_of(q), order(tables[n]), layout) for n in sizes]
    x = np.concatenate([p[0] for p in parts])
    offs = np.cumsum([0] + [1 << n for n in logns])
    dx, dy = DevBuf.from_array(ctx, order(x)), DevBuf(ctx, x.nbytes)
    engine = bn.Batch(ctx, plans)
    engine.run_dev(bn.Batch.jobs([dx.addr + 16 * int(o) for o in offs[:-1]], [dy.addr + 16 * int(o) for o in offs[:-1]],
                                 [sizes.index(n) for n in logns]))
    assert engine.status() == bn.OK
    want = np.concatenate([C.oracle_ntt(p[0], tables[n], n, q, mu_of(q)) for n, p in zip(logns, parts)])
    assert np.array_equal(order(dy.to_array()), want)
    engine.close()
    for p in plans:
        p.close()
    dx.free()
    dy.free()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["edges", "sparse", "ternary"])
@pytest.mark.parametrize("logn", [3, 4, 5, 6, 7, 8, 9, 10, 11, 13, 16, 17])
@pytest.mark.parametrize("elems", [1 << 17, 1 << 18, 1 << 21], ids=["lone", "few", "many"])
def test_every_launch_size_matches_oracle(ctx, kind, logn, elems):
    """The plan kernels of each launch size (up to 2^17 elements, below 2^21, above), with a ragged last
    tile: a few distinct transforms repeated, so the oracle computes only those."""
    q = C.Q_NTT
    rows = max(1, min(7, 4096 >> logn))
    x, t = values(kind, q, logn, rows)
    batch = elems >> logn if elems == 1 << 17 else (elems >> logn) + 3
    at = (np.arange(batch) % rows)[:, None] * (1 << logn) + np.arange(1 << logn)
    plan = bn.Plan(ctx, logn, q, mu_of(q), t)
    dx, dy = DevBuf.from_array(ctx, x[at.reshape(-1)]), DevBuf(ctx, batch * 16 << logn)
    bn.check(bn.lib().bntt_ntt_forward_dev(plan.handle, dy.ptr, dx.ptr, batch))
    want = C.oracle_ntt(x, t, logn, q, mu_of(q), form=1, threads=8)
    assert np.array_equal(dy.to_array(), want[at.reshape(-1)])
    dx.free()
    dy.free()
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("logn", [1, 2, 3, 5, 6, 7, 8, 9, 10, 11, 13, 16])
@pytest.mark.parametrize("elems", [1 << 17, 1 << 18, 1 << 21], ids=["lone", "few", "many"])
def test_inverse_of_every_launch_size(ctx, logn, elems):
    """The inverse kernels of each launch size on special values, against the oracle."""
    q = Q_NC
    rows = max(1, min(7, 4096 >> logn))
    y = values("ternary", q, logn, rows)[0]
    y[y.shape[0] // 2:] = C.uniform_pairs(5, y.shape[0] - y.shape[0] // 2, q)
    t = C.uniform_pairs(6 + logn, 1 << logn, q)
    batch = elems >> logn if elems == 1 << 17 else (elems >> logn) + 3
    at = (np.arange(batch) % rows)[:, None] * (1 << logn) + np.arange(1 << logn)
    plan = bn.Plan(ctx, logn, q, mu_of(q), t)
    dy, dx = DevBuf.from_array(ctx, y[at.reshape(-1)]), DevBuf(ctx, batch * 16 << logn)
    bn.check(bn.lib().bntt_ntt_inverse_dev(plan.handle, dx.ptr, dy.ptr, batch))
    want = C.oracle_ntt_inverse(y, t, logn, q, mu_of(q))
    assert np.array_equal(dx.to_array(), want[at.reshape(-1)])
    dx.free()
    dy.free()
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("logn", [9, 10, 13])   # inverse table built on the host, on the device
@pytest.mark.parametrize("entry", [1, 2, "last"])
def test_tables_without_an_inverse_are_refused(logn, entry):
    """A zero twiddle anywhere, and a composite modulus, are refused whichever
    side builds the inverse table; entry 0, which no stage reads, may be 0."""
    ctx = bn.Context(0)
    n = 1 << logn
    d = DevBuf.from_array(ctx, C.uniform_pairs(5, n, C.Q_NTT))
    t = C.uniform_pairs(6, n, C.Q_NTT)
    t[0] = 0
    good = bn.Plan(ctx, logn, C.Q_NTT, C.MU_NTT, t)
    assert bn.lib().bntt_ntt_inverse_dev(good.handle, d.ptr, d.ptr, 1) == bn.OK
    want = C.oracle_ntt_inverse(C.uniform_pairs(5, n, C.Q_NTT), t, logn)
    assert np.array_equal(d.to_array(), want)
    t[n - 1 if entry == "last" else entry] = 0
    zero = bn.Plan(ctx, logn, C.Q_NTT, C.MU_NTT, t)
    assert bn.lib().bntt_ntt_inverse_dev(zero.handle, d.ptr, d.ptr, 1) == bn.EINVAL
    assert b"no inverse" in bn.lib().bntt_last_error()
    q = (1 << 124) - 721                            # a multiple of 3
    assert q % 3 == 0
    comp = bn.Plan(ctx, logn, q, mu_of(q), C.uniform_pairs(7, n, q))
    assert bn.lib().bntt_ntt_inverse_dev(comp.handle, d.ptr, d.ptr, 1) == bn.EINVAL
    assert np.array_equal(d.to_array(), want)       # nothing was written
    for o in (good, zero, comp):
        o.close()
    d.free()
    ctx.close()
