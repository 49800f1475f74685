"""ADI wells whose lines fit a warp's registers (up to 1024 positions) next to
wells with longer lines: batched and alone, a well runs the same operations in
the same order, so its field is the same bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wells", [
    # one small well: one line per warp
    [(33, 31, True, False)],
    # 1 to 32 chunks, ragged ends, lines that do not fill a CTA
    [(1, 1, False, False), (5, 1023, False, True), (32, 33, True, True), (96, 97, False, False),
     (1024, 36, True, False), (511, 513, False, False), (255, 64, False, True)],
    # either side or both past 1024
    [(1025, 40, False, False), (40, 1025, True, True), (1030, 1029, False, True), (1024, 1024, False, False)],
    # enough wells for several lines per warp
    [(63 + i, 130 - i, i % 2 == 0, i % 3 == 0) for i in range(60)],
    # around the numbers of lines at which a single grid leaves the warp per line
    # (a wave of 1216) and comes back to it (half of the next)
    [(520, 1215, False, True), (520, 1216, True, False), (1024, 1220, False, False), (1217, 993, True, True),
     (544, 1823, False, False), (1824, 600, False, True), (512, 1300, False, False)],
], ids=["one", "chunks", "long", "many", "many-lines"])
def test_line_wells_equal_single_grids(hal, wells):
    rng = np.random.default_rng(len(wells))
    desc = [dict(xDim=x, yDim=y, kind="adi", diffRate=0.5 + i % 7, decay=0.01 * (i % 2), wrapX=wx, wrapY=wy,
                 maxAgents=0) for i, (x, y, wx, wy) in enumerate(wells)]
    f = [rng.random(d["xDim"] * d["yDim"]).astype(np.float32) for d in desc]
    s = [(rng.random(a.size) * 0.01).astype(np.float32) if i % 2 else None for i, a in enumerate(f)]
    with hal.Wells(desc) as b:
        for i, a in enumerate(f):
            b.set_field(i, a)
            if s[i] is not None:
                b.set_source(i, s[i])
        b.run_ticks(3, 1.0, 0.1)
        got = [b.get_field(i) for i in range(len(desc))]
    for i, d in enumerate(desc):
        with hal.Adi(d["xDim"], d["yDim"]) as h:
            h.set_field(f[i])
            if s[i] is not None:
                h.set_source(s[i])
            h.run_ticks(3, d["diffRate"], d["decay"], d["wrapX"], d["wrapY"])
            assert np.array_equal(got[i], h.get_field()), (i, d)
