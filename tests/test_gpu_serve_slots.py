"""The step loops of a chunk by the slots they cover: solves in the first, a
middle and the last slot, few and all of them, retiring one after the other --
each equal, bit for bit, to the same solve on its own."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("slots,steps", [(1, [5]), (4, [3, 9, 1]), (5, [2, 7, 4, 1, 12]), (16, [4] * 13 + [9, 1])])
def test_solves_do_not_depend_on_their_slots(built_lib, precision, slots, steps):
    from exactclosure_gb300 import navierstokes as NS
    from exactclosure_gb300.serving import Server

    n = 32
    sv = Server(precision=precision, autotune=False, slots_per_chunk=slots)
    for _ in range(2):  # the second pass meets loops that are there already
        ids = [sv.submit(n, 1 / 500, k, seed=i, keep_field=True) for i, k in enumerate(steps)]
        sv.drain()
        got = {r["id"]: r for r in sv.poll()}
        for i, k in enumerate(steps):
            cs = NS.Case(n, 1.0, 1 / 500, 0.3, precision=precision)
            cs.init_random(4.0, 1.0, i)
            cs.step(k)
            assert (cs.velocity() == got[ids[i]]["field"]).all()
            assert got[ids[i]]["sim_time"] == cs.time()[0]
            cs.close()
    sv.close()
