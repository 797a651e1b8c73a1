"""The tile-wise update where its blocks hold several bytes of the change
bitmaps (1216 blocks, 256 bytes a pass each): some bytes a block with
substates of every type, and more than one pass with 32 byte substates.  Each
step changes some of the tiles of each substate, and some cells of those, by
amounts that depend on the current layer, so that a tile left out or copied
from the wrong substate shows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _body(kinds):
    lines = ["const int tile = (i / 8) * 13 + (j / 32) * 7, cell = i * 31 + j * 17;"]
    for k, t in enumerate(kinds):
        lines.append(f"if ((tile + {k}) % 5 < 2 && (cell + {5 * k}) % 7 == 0) "
                     f"calSet2D{t}(ca, Q.s{k}, i, j, calGet2D{t}(ca, Q.s{k}, i, j) + (i + j) % 9 + 1);")
    return "\n".join(lines)


@pytest.mark.parametrize("rows,cols,kinds", [(2200, 2300, "birb"), (4480, 4470, "b" * 32)])
def test_many_bitmap_bytes_a_block(rows, cols, kinds):
    import opencal_gb300 as cal
    from opencal_gb300 import program as P
    cal.build()
    tiles = -(-rows // 8) * -(-cols // 32)
    items = len(kinds) * 4 * -(-tiles // 32)
    assert items > (1216 * 256 if len(kinds) == 32 else 1216)
    prog = P.Program(f"lists{len(kinds)}").substates(**{f"s{k}": t for k, t in enumerate(kinds)})
    lib = prog.process("rule", _body(kinds)).build()
    steps = 3
    with P.Model2D(rows, cols, P.CAL_VON_NEUMANN_NEIGHBORHOOD_2D, P.CAL_SPACE_FLAT) as model:
        subs = [model.add_substate(t) for t in kinds]
        lib.bind(**{f"s{k}": s for k, s in enumerate(subs)})
        model.add_process(lib.process("rule"))
        for s in subs:
            model.init(s, 0)
        run = P.Run2D(model, 1, steps, graph=True)
        run.run()
        i, j = np.arange(rows)[:, None], np.arange(cols)[None, :]
        tile, cell = (((i // 8) * 13 + (j // 32) * 7) % 5).astype(np.int8), ((i * 31 + j * 17) % 7).astype(np.int8)
        add = (steps * ((i + j) % 9 + 1)).astype(np.int8)
        for k, s in enumerate(subs):
            in_tile = np.array([(t + k) % 5 < 2 for t in range(5)])[tile]
            in_cell = np.array([(c + 5 * k) % 7 == 0 for c in range(7)])[cell]
            assert np.array_equal(model.read(s), add * (in_tile & in_cell)), k
        run.close()
