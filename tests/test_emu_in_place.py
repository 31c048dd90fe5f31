"""In-place tiles (csrc/sk_modes.h SK_IN_PLACE) on the CPU harness against the
FP64 oracle: every tile mode and operation, staged and direct input, two to
four passes, odd radices, partial tiles, an odd number of real rows and
column counts that are no multiple of the tile.  Shared memory starts as NaN,
so a slot read before it was written shows.  Tolerance: the library's
rel-L2 bar of 1e-6."""
import json

import pytest

from oracle import oracle as O
from tests.fftcase import emu_run, random_input

F, I = O.FORWARD, O.INVERSE
CASES = [
    (O.C2C, F, [1320], 3), (O.C2C, F, [1320], 7), (O.C2C, I, [1320], 1), (O.C2C, I, [1320], 5),
    (O.C2C, F, [1155], 5), (O.C2C, I, [1155], 2),
    (O.C2C, I, [390, 8], 2), (O.C2C, I, [390, 7], 3), (O.C2C, F, [390, 7], 2), (O.C2C, F, [390, 1], 3),
    (O.R2C, F, [780], 3), (O.R2C, I, [780], 4), (O.C2R, I, [780], 5), (O.C2R, F, [780], 3),
    (O.R2C, F, [715], 4), (O.R2C, I, [715], 7), (O.C2R, I, [715], 8), (O.C2R, F, [715], 5),
]


@pytest.mark.parametrize("op,direction,sizes,batch", CASES)
def test_in_place_tiles(emu, op, direction, sizes, batch):
    x = random_input(op, sizes, batch, seed=sum(sizes) + batch)
    rc, out, desc = emu_run(emu, op, direction, sizes, batch, x)
    assert rc == 0, desc
    steps = json.loads(desc)["steps"]
    assert any(s.get("sk_cfg", [0] * 9)[8] & 16 for s in steps), desc[:400]
    assert O.rel_l2(out, O.fp64(op, direction, x, sizes)) <= 1e-6
