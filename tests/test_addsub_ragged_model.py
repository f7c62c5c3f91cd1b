"""CPU model of the ragged add/sub kernel's copies (addsub.cu): a CTA's tiles are
copied into two stages, two ahead.  Wherever a wait runs out, the stages that it
waits for again before it leaves are those with a copy under way, at the phases
that those copies complete."""
import pytest


@pytest.mark.parametrize("grid", [1, 2, 3])
@pytest.mark.parametrize("ntiles", range(1, 12))
def test_leaving_waits_for_every_copy(grid, ntiles):
    for block in range(min(grid, ntiles)):
        mine = list(range(block, ntiles, grid))
        for fails in range(len(mine)):
            asked, phase = {}, [0, 0]              # tile -> (stage, phase) of copies asked for

            def fetch(tile, st):
                asked[tile] = (st, phase[st] & 1)
                phase[st] += 1

            fetch(block, 0)
            if block + grid < ntiles:
                fetch(block + grid, 1)
            for it, tile in enumerate(mine[:fails + 1]):
                st = it & 1
                assert asked[tile] == (st, it >> 1 & 1)
                if it == fails:
                    again = {(st, it >> 1 & 1)}
                    if tile + grid < ntiles:
                        again.add((st ^ 1, it + 1 >> 1 & 1))
                    assert again == set(asked.values())
                    break
                del asked[tile]                    # arrived; the stage is free after the tile
                if tile + 2 * grid < ntiles:
                    fetch(tile + 2 * grid, st)
