"""The resident solve's verdict words (csrc/resident.cuh), on the CPU.

At each reduction the scalar warp writes a verdict (go on / leave), the block meets
at a barrier, and every row warp reads the verdict and goes on or leaves.  Once a poll
has run out the scalar warp does not wait for the row warps' contributions any more:
all interleavings of one scalar and two row warps are walked here, with the
reductions in the order and the verdict words in the places that the source gives
them, for every point at which polls may give up.  All row warps have to take the
same decision (one that leaves alone strands the others at the row warps' barrier,
which has no limit), and the leave has to be seen."""
import pathlib
import re

import pytest

SRC = pathlib.Path(__file__).resolve().parent.parent / "2clowns-3d_gb300" / "csrc" / "resident.cuh"


def _between(text, start, end):
    at = text.index(start)
    return text[at:text.index(end, at)]


def _orders():
    """Reductions in program order: a plain and a mixed solve of a few iterations."""
    text = SRC.read_text()
    reds = lambda body: [int(v) for v in re.findall(r"totals<\d>\((\d),", body)]
    loop = reds(_between(text, "void iterate(", "void finish("))
    plain = reds(_between(text, "k_res_plain(const", "k_res_mixed(const"))
    mixed = reds(text[text.index("k_res_mixed(const"):])
    assert loop == [0, 1, 2] and len(plain) == 2 and len(mixed) == 3
    sweeps = []
    for leave in (1, 2, 3):                    # an inner solve may end at any reduction of an iteration
        sweeps += mixed[1:] + loop + loop[:leave]
    return {"plain": plain + 2 * loop, "mixed": mixed[:1] + sweeps + mixed[1:2]}


def _word(red):
    """The verdict word of a reduction, as `totals` writes and reads it."""
    body = _between(SRC.read_text(), "bool totals(", "// The iterations of one")
    writes, = re.findall(r"sh\.stop(\[red\])? =[^=]", body)
    reads, = re.findall(r"sh\.stop(\[red\])? ==", body)
    assert writes == reads
    return red if writes else 0


def _split(order, gave_up, words):
    """Whether some interleaving makes the row warps part: verdicts from reduction
    `gave_up` on say leave, and the scalar warp waits for nobody from then on."""
    last = len(order) - 1
    # scalar: (reduction, written); rows: (reduction, 0 before the barrier / 1 to read / 2 left)
    start = ((0, False), ((0, 0), (0, 0)), tuple(0 for _ in range(words)))
    seen, todo = {start}, [start]
    while todo:
        (k, written), rows, mem = todo.pop()
        nxt = []
        if k <= last and not written and (k >= gave_up or all(r == (k, 0) for r in rows)):
            m = list(mem)
            m[_WORD[order[k]]] = int(k >= gave_up)
            nxt.append(((k, True), rows, tuple(m)))
        if written and all(r == (k, 0) for r in rows):          # the block's barrier
            nxt.append(((k + 1, False) if k < gave_up else (last + 1, False), tuple((k, 1) for _ in rows), mem))
            if k < last and k >= gave_up - 1:                   # polls give up at once: the next verdict may come
                nxt.append(((k + 1, False), tuple((k, 1) for _ in rows), mem))
        for i, (rk, ph) in enumerate(rows):
            if ph != 1:
                continue
            leave = mem[_WORD[order[rk]]]
            if leave != int(rk >= gave_up):
                return True
            new = list(rows)
            new[i] = (rk, 2) if leave or rk == last else (rk + 1, 0)
            nxt.append(((k, written), tuple(new), mem))
        for st in nxt:
            if st not in seen:
                seen.add(st)
                todo.append(st)
    return False


_WORD = {}


@pytest.mark.parametrize("kind", ["plain", "mixed"])
def test_row_warps_take_one_decision(kind):
    order = _orders()[kind]
    _WORD.update({r: _word(r) for r in set(order)})
    for gave_up in range(1, len(order)):
        assert not _split(order, gave_up, max(_WORD.values()) + 1), (kind, gave_up)


def test_a_single_word_would_part_them():
    """The walk sees the fault it is for."""
    _WORD.update({r: 0 for r in range(5)})
    assert _split(_orders()["plain"], 1, 1)
