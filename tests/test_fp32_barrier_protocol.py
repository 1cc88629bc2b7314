"""A model of the mbarrier protocol of the fp32 tcgen05 kernels (csrc/fwd_f32_tc5.cu, csrc/bwd_f32_tc5.cu), run under random
interleavings on the CPU.

One CTA works on the tiles of one item.  Roles: the TMA producer, one issuing warp, two elementwise groups, and in the launch that
owns keys a warp that stages the queries' statistics.  The producer fills one ring of units in the order in which the issuing warp
asks for them: the scores of tile t + 1, then the outputs of tile t (with a single score buffer the scores of tile t).  The launch
that owns keys keeps all units of a tile's Q until S is formed and asks for them in another order than they lie in (`held`).
Barriers, with the kernels' names: full / empty per unit; s_full, p_full per score buffer; acc_full / acc_free, one phase per
piece of a tile's outputs; meet (forward); stat_full (launch that owns keys).  The engine is the one of the other models
(tests/test_pipe128_barrier_protocol.py).
"""
import pytest

from tests.test_fused64_barrier_protocol import in_order
from tests.test_pipe128_barrier_protocol import World


def run_fp32(seed, n_tiles, stages, scores, pieces, buffers=2, held=0, meet=False, stats=False):
    """scores, pieces: units of a tile's scores (of which the first `held` are kept), and of each piece of its outputs."""
    w = World(seed)
    full, empty = [w.bar(1) for _ in range(stages)], [w.bar(1) for _ in range(stages)]
    s_full, p_full, stat_full = ([w.bar(n), w.bar(n)] for n in (1, 2, 1))
    acc_full, acc_free, meets = w.bar(1), w.bar(2), w.bar(2)
    order = [("s", 0)]
    for t in range(n_tiles):
        order += [("s", t + 1), ("o", t)] if buffers == 2 else [("o", t), ("s", t + 1)]
    order = [(what, t) for what, t in order if t < n_tiles]

    def producer():
        n = 0
        for what, t in order:
            for _ in range(scores if what == "s" else sum(pieces)):
                yield from w.wait(empty[n % stages], ((n // stages) & 1) ^ 1, ("free", n - stages) if n >= stages else None)
                w.later(lambda n=n: (w.events.add(("unit", n)), full[n % stages].arrive()))
                n += 1
                yield

    def free(n):
        w.later(lambda: (w.events.add(("free", n)), empty[n % stages].arrive()))

    def issuer():
        n = piece = 0

        def loaded(m):
            return w.wait(full[m % stages], (m // stages) & 1, ("unit", m))

        for what, t in order:
            if what == "s":
                assert t < buffers or ("p", t - buffers) in w.events  # S is formed over the parts of P, whose products were issued before
                slices = held // 3
                for p in (2, 1, 0) if held else ():
                    for s in range(slices):
                        yield from loaded(n + 3 * s + 2 - p)
                        for x in range(3) if p == 0 else ():
                            free(n + 3 * s + x)
                        yield
                n += held
                for i in range(scores - held):
                    yield from loaded(n)
                    free(n)
                    if i == scores - held - 1:
                        w.later(lambda t=t: (w.events.add(("s", t)), s_full[t % buffers].arrive()))
                    n += 1
                    yield
            else:
                yield from w.wait(p_full[t % buffers], (t // buffers) & 1, ("p", t))
                for units in pieces:
                    if piece > 0:
                        yield from w.wait(acc_free, (piece - 1) & 1, ("read", piece - 1))
                    for i in range(units):
                        yield from loaded(n)
                        free(n)
                        if i == units - 1:
                            w.later(lambda k=piece: (w.events.add(("acc", k)), acc_full.arrive()))
                        n += 1
                        yield
                    piece += 1

    def elementwise():
        piece = 0
        for t in range(n_tiles):
            if stats:
                yield from w.wait(stat_full[t & 1], (t >> 1) & 1, ("stat", t))
            yield from w.wait(s_full[t % buffers], (t // buffers) & 1, ("s", t))
            if meet:
                w.tally(("m", t), 2, ("met", t))
                meets.arrive()
                yield from w.wait(meets, t & 1, ("met", t))
            w.tally(("pt", t), 2, ("p", t))
            p_full[t % buffers].arrive()
            yield
            for _ in pieces:
                yield from w.wait(acc_full, piece & 1, ("acc", piece))
                w.tally(("rt", piece), 2, ("read", piece))
                acc_free.arrive()
                piece += 1
                yield

    def statistics():
        for t in range(n_tiles if stats else 0):
            if t >= 2:
                yield from w.wait(p_full[t & 1], ((t >> 1) - 1) & 1, ("p", t - 2))
            w.events.add(("stat", t))
            stat_full[t & 1].arrive()
            yield

    agents = [producer(), in_order(w, issuer()), elementwise(), elementwise(), statistics()]
    return w.run(agents, ["producer", "issuer", "elementwise 0", "elementwise 1", "statistics"])


@pytest.mark.parametrize("n_tiles", [1, 2, 3, 8])
@pytest.mark.parametrize("kernel", [
    dict(stages=12, scores=3, pieces=[3], meet=True), dict(stages=8, scores=3, pieces=[3], meet=True),  # forward, D <= 64
    dict(stages=8, scores=6, pieces=[3], meet=True), dict(stages=4, scores=6, pieces=[3, 6], meet=True),  # ... D = 128
    dict(stages=4, scores=6, pieces=[3, 3], meet=True),
    dict(stages=16, scores=6, pieces=[3]), dict(stages=12, scores=12, pieces=[6]),  # own queries, through O
    dict(stages=10, scores=6, pieces=[3]), dict(stages=4, scores=12, pieces=[6], buffers=1),  # ... through tO
    dict(stages=16, scores=6, pieces=[6], held=3, stats=True), dict(stages=8, scores=12, pieces=[6, 6], held=6, stats=True),  # own keys
], ids=str)
def test_fp32_protocol_has_no_deadlock_and_no_premature_pass(kernel, n_tiles):
    for seed in range(8):
        assert run_fp32(seed, n_tiles, **kernel) == "ok", (kernel, n_tiles, seed)
