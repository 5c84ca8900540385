"""The order of the prompt attention kernel's hand-overs between its roles, as a graph of who waits for whom (the constants are the kernel's)."""
import itertools
import re
from pathlib import Path

import pytest

import cubic_serve_b200

SOURCE = (Path(cubic_serve_b200.__file__).parent / "csrc" / "paged_prefill.cu").read_text()


def _constant(name):
    value = re.search(rf"constexpr int {name} = ([^;]+);", SOURCE).group(1)
    return eval(re.sub(r"kPf\w+", lambda m: str(_constant(m.group(0))), value), {})      # noqa: S307 (sums of integers)


def _waits(taking_part, raw):
    """event -> events before it, for steps in which ``taking_part[step]`` tiles see something."""
    before = {}

    def after(event, *others):
        before.setdefault(event, set()).update(o for o in others if o is not None)

    last_read = {}
    for g, tiles in enumerate(taking_part):
        step = lambda what, back=0: (what, g - back) if g >= back else None  # noqa: E731
        after(("copied", g), step("copied", 1), step("k converted", raw), step("v converted", raw))       # raw_free
        after(("k note", g), ("copied", g), step("k converted", 1), step("k free", 2))
        after(("k converted", g), ("k note", g))
        after(("v note", g), ("copied", g), step("v converted", 1), step("v free", 2))
        after(("v converted", g), ("v note", g))
        after(("k free", g), ("k converted", g), step("k free", 1))
        after(("v free", g), ("v converted", g), step("v free", 1))
        for t in tiles:
            before_it = last_read.get(t)
            after(("scores", g, t), ("k converted", g), before_it and ("scores read", *before_it))         # k_full, s_free
            after(("k free", g), ("scores", g, t))
            after(("scores read", g, t), ("scores", g, t), before_it and ("probabilities", *before_it))    # s_full; a warp's own order
            after(("notes read", g, t), ("scores read", g, t), ("k note", g), ("v note", g))
            after(("probabilities", g, t), ("notes read", g, t))
            after(("v free", g), ("probabilities", g, t))                                                  # p_full, the product
            last_read[t] = (g, t)
    return before


def _is_before(before, early, late):
    seen, todo = set(), [late]
    while todo:
        e = todo.pop()
        if e == early:
            return True
        if e not in seen:
            seen.add(e)
            todo += before.get(e, ())
    return False


def _in_order(raw, notes):
    for pattern in itertools.product(((0,), (1,), (0, 1)), repeat=7):
        before = _waits(pattern, raw)
        for g, tiles in enumerate(pattern[:len(pattern) - notes]):
            for t, note in itertools.product(tiles, ("k note", "v note")):
                if not _is_before(before, ("notes read", g, t), (note, g + notes)):
                    return False
    return True


def test_notes_are_written_behind_every_read():
    """Whichever tiles take part in which steps: no note of a step is written before the tiles have read the one in its place."""
    raw, notes = _constant("kPfRaw"), _constant("kPfNotes")
    assert _in_order(raw, notes)


@pytest.mark.parametrize("notes", [2, 3, 4])
def test_fewer_notes_would_not_do(notes):
    assert not _in_order(3, notes)
