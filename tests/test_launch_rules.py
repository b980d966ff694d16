"""Rules by which launches are cut and placed, on the CPU."""
import re

import pytest

from flambeau_b200.kernels.build import CSRC
from flambeau_b200.kernels.library import lib

SMS = 148


def test_stretches_of_decoded_tokens_over_latents_fill_whole_rounds():
    """Rounds of CTAs times the tiles of a stretch stay near what an even share of all tiles would be; every stretch has tiles."""
    for tiles in (100, 125, 250, 512):
        for pairs in range(1, 257):
            s = lib().fb_attention_tc_stretches(pairs, tiles, 64, SMS)
            per = max(4, -(-tiles // s))
            assert s >= 3 and (s - 1) * per < tiles
            rounds = -(-pairs * s // SMS)
            # half a tile of rounding up a stretch, three tiles a CTA for what it costs to start one
            assert rounds * per <= 1.2 * pairs * tiles / SMS + 3 * rounds + per or rounds == 1, (pairs, tiles, s)
    assert lib().fb_attention_tc_stretches(38, 125, 64, SMS) * 38 % SMS > SMS // 2, "a last round that is nearly empty"
    for tiles in (1, 3, 4, 5, 13):                       # few tiles: never a stretch without one
        for pairs in (1, 8, 64, 300):
            s = lib().fb_attention_tc_stretches(pairs, tiles, 64, SMS)
            assert 1 <= s <= -(-tiles // 4)
    assert lib().fb_attention_tc_stretches(8, 125, 0, SMS) == 0 and lib().fb_attention_tc_stretches(8, 125, 2, SMS) == 2


def test_rows_of_a_grouped_products_tiles():
    """Tiles of 32 only for the kernel that joins them; the one-SM kernel has tiles of its own sizes."""
    from flambeau_b200.kernels import ops
    try:
        ops.set_gemm_pair(True)
        assert [ops.grouped_tile(n, 4, True) for n in (1, 64, 65, 767, 768, 9999)] == [16, 16, 32, 32, 32, 32]
        assert [ops.grouped_tile(n, 4, False) for n in (64, 65, 9999)] == [16, 64, 64]
        ops.set_gemm_pair(False)
        assert [ops.grouped_tile(n, 4, True) for n in (1, 64, 65, 767, 768, 9999)] == [16, 16, 64, 64, 128, 128]
        assert [ops.grouped_tile(n, 4, False) for n in (64, 65, 9999)] == [16, 64, 64]
    finally:
        ops.set_gemm_pair(True)


def kernels(path):
    """(name, source) of every kernel of a file."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    for m in re.finditer(r"__global__[^;{]*?(\w+)\(const __grid_constant__[^{]*\{", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield m.group(1), text[m.end():end]


TAKE_TENSOR_MEMORY = sorted(p.stem for p in CSRC.glob("*.cu") if re.search(r"tmem_alloc\(|tcgen05\.alloc", p.read_text()))


@pytest.mark.parametrize("file", TAKE_TENSOR_MEMORY)
def test_dependents_come_behind_tensor_memory(file):
    """A kernel placed early that got its columns first would wait for this one's end, and this one for its columns."""
    found = 0
    for name, source in kernels(CSRC / f"{file}.cu"):
        alloc = re.search(r"tmem_alloc\(|tcgen05\.alloc", source)
        if alloc:
            found += 1
            lets_in = source.index("fb_pdl_launch_dependents()")
            assert alloc.start() < lets_in and "__syncthreads()" in source[alloc.start():lets_in], name
    assert found == 1
