"""FP64 served solves at grids where a batch gives the CTAs of the right-hand
side's sweep more planes than a single field does (csrc/rhs.cu): the bits of a
solve alone, of a case and of the same solve among others."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 96])
def test_fp64_solves_do_not_depend_on_the_batch(built_lib, n):
    from exactclosure_gb300 import navierstokes as NS
    from exactclosure_gb300.serving import Server

    steps, ref = 4, {}
    for seed in range(8):
        cs = NS.Case(n, 1.0, 1 / 2000, 0.3)
        cs.init_random(4.0, 1.0, seed)
        cs.step(steps)
        ref[seed] = cs.velocity()
        cs.close()
    for slots in (1, 3, 8):
        sv = Server(precision=0, autotune=False, slots_per_chunk=slots)
        ids = {sv.submit(n, 1 / 2000, steps, seed=s, keep_field=True): s for s in range(slots)}
        sv.drain()
        for r in sv.poll():
            assert (r["field"] == ref[ids[r["id"]]]).all(), (slots, ids[r["id"]])
        sv.close()
