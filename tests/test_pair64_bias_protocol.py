"""The head-dimension-64 forward with a bias (csrc/fwd_tc5_pair64.cu, MK = 2): K and V have rings of two stages each and every query
tile a bias tile of its own.  A model of its barriers under random interleavings, in the manner of test_pair64_barrier_protocol.py."""
import pytest

from tests.test_fused64_barrier_protocol import in_order
from tests.test_pipe128_barrier_protocol import World

STAGES = 2


def run(items, seed, grow_prob=0.3, wait_for_v=True):
    """items[k]: (key tiles, query tiles in use as bits); a query tile that starts behind the last row uses none.  wait_for_v: without it an
    issuer releases a stage of V that it does not use before its turn."""
    w = World(seed)
    bars = lambda n, c: [w.bar(c) for _ in range(n)]  # noqa: E731
    q_full, q_empty = w.bar(1), w.bar(2)
    k_full, k_empty, v_full, v_empty = bars(STAGES, 1), bars(STAGES, 2), bars(STAGES, 1), bars(STAGES, 2)
    b_full, b_empty = bars(2, 1), bars(2, 1)
    s_full, s_free, p_full, pv_done, o_free = (bars(2, 1) for _ in range(5))

    def producer():
        g, nb = 0, [0, 0]
        for kact, (n, used) in enumerate(items):
            if kact:
                yield from w.wait(q_empty, (kact - 1) & 1, ("q_released", kact - 1))
            w.later(lambda kact=kact: (w.events.add(("q", kact)), q_full.arrive()))
            for _ in range(n):
                st, par = g % STAGES, ((g // STAGES) & 1) ^ 1
                yield from w.wait(k_empty[st], par, ("k_free", g - STAGES) if g >= STAGES else None)
                w.later(lambda g=g, st=st: (w.events.add(("k", g)), k_full[st].arrive()))
                for x in range(2):
                    if used & (1 << x):
                        yield from w.wait(b_empty[x], (nb[x] & 1) ^ 1, ("b_read", x, nb[x] - 1) if nb[x] else None)
                        w.later(lambda x=x, t=nb[x]: (w.events.add(("b", x, t)), b_full[x].arrive()))
                        nb[x] += 1
                yield from w.wait(v_empty[st], par, ("v_free", g - STAGES) if g >= STAGES else None)
                w.later(lambda g=g, st=st: (w.events.add(("v", g)), v_full[st].arrive()))
                g += 1
                yield

    def issuer(X):
        g, T, kx = 0, 0, 0
        for kact, (n, used) in enumerate(items):
            yield from w.wait(q_full, kact & 1, ("q", kact))
            pend, first = None, True

            def issue_pv(p):
                pg, pT, pfirst = p
                yield from w.wait(p_full[X], pT & 1, ("p", X, pT))
                yield from w.wait(v_full[pg % STAGES], (pg // STAGES) & 1, ("v", pg))
                if pfirst and kx > 0:
                    yield from w.wait(o_free[X], (kx - 1) & 1, ("o_read", X, kx - 1))
                w.later(lambda: (w.tally(("vf", pg), 2, ("v_free", pg)), v_empty[pg % STAGES].arrive(),
                                 w.events.add(("pv", X, pT)), pv_done[X].arrive()))
                yield

            for j in range(n):
                st = g % STAGES
                yield from w.wait(k_full[st], (g // STAGES) & 1, ("k", g))
                if used & (1 << X):
                    if T > 0:
                        yield from w.wait(s_free[X], (T - 1) & 1, ("s_read", X, T - 1))

                    def scores_done(T=T, g=g, st=st, last_one=(j == n - 1), kact=kact):
                        w.events.add(("s", X, T))
                        s_full[X].arrive()
                        w.tally(("kf", g), 2, ("k_free", g))
                        k_empty[st].arrive()
                        if last_one:
                            w.tally(("qr", kact), 2, ("q_released", kact))
                            q_empty.arrive()

                    w.later(scores_done)
                    yield
                    if pend is not None:
                        yield from issue_pv(pend)
                    pend, first = (g, T, first), False
                    T += 1
                else:
                    if wait_for_v:
                        yield from w.wait(v_full[st], (g // STAGES) & 1, ("v", g))
                    w.tally(("kf", g), 2, ("k_free", g))
                    k_empty[st].arrive()
                    w.tally(("vf", g), 2, ("v_free", g))
                    v_empty[st].arrive()
                    yield
                g += 1
            if pend is not None:
                yield from issue_pv(pend)
            if not first:
                kx += 1
            else:
                w.tally(("qr", kact), 2, ("q_released", kact))
                q_empty.arrive()
            yield

    def softmax(X):
        T, kx = 0, 0
        for n, used in items:
            if not used & (1 << X):
                yield
                continue
            for u in range(n):
                yield from w.wait(s_full[X], T & 1, ("s", X, T))
                w.events.add(("s_read", X, T))
                s_free[X].arrive()
                yield
                yield from w.wait(b_full[X], T & 1, ("b", X, T))
                w.events.add(("b_read", X, T))
                b_empty[X].arrive()
                yield
                if T > 0:
                    if u > 0 and w.rnd.random() < grow_prob:
                        yield from w.wait(pv_done[X], (T - 1) & 1, ("pv", X, T - 1))
                    yield from w.wait(pv_done[X], (T - 1) & 1, ("pv", X, T - 1))
                w.events.add(("p", X, T))
                p_full[X].arrive()
                T += 1
                yield
            yield from w.wait(pv_done[X], (T - 1) & 1, ("pv", X, T - 1))
            w.events.add(("o_read", X, kx))
            o_free[X].arrive()
            kx += 1
            yield

    agents = [producer(), in_order(w, issuer(0)), in_order(w, issuer(1)), softmax(0), softmax(1)]
    return w.run(agents, ["producer", "issuer0", "issuer1", "softmax0", "softmax1"])


@pytest.mark.parametrize("items", [[(1, 3)], [(7, 3)], [(5, 3), (2, 1), (1, 3)], [(4, 1), (4, 3), (4, 1), (1, 1)], [(9, 3), (9, 1)]], ids=str)
def test_bias_protocol(items):
    for seed in range(40):
        assert run(items, seed) == "ok", (items, seed)
    assert run(items, 99, grow_prob=1.0) == "ok"


def test_the_model_shows_a_stage_released_before_its_turn():
    found = 0
    for seed in range(40):
        try:
            found += run([(9, 1), (9, 3)], seed, wait_for_v=False) != "ok"
        except AssertionError:
            found += 1
    assert found
