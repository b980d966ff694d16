"""Rules by which launches are cut, on the CPU."""
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
