"""Which kernel a latent prompt step takes: steps timed in all of them, of prompts of about the same context each."""
import pytest

from cuteafd_b200.ops import native

# chunks of key columns, of rotated ones, of value columns; heads; rows of the sequences; us in the one-tile kernel, with one tile per CTA and with pairs in the paired one
STEPS = [
    ((1, 0, 1), 12, [2048], (35.8, 33.8, 39.9)), ((1, 0, 1), 48, [300], (50.5, 49.5, 58.4)), ((1, 0, 1), 16, [889, 230], (71.2, 70.6, 81.3)), ((1, 0, 1), 128, [2048], (564, 550, 349)),
    ((1, 1, 2), 12, [2048], (37.9, 44.1, 49.6)), ((1, 1, 2), 12, [1024], (50.3, 58.4, 66.2)), ((1, 1, 2), 48, [300], (55.0, 62.5, 70.6)), ((1, 1, 2), 48, [100] * 12, (54.3, 62.5, 62.5)),
    ((1, 1, 2), 128, [2048], (604, 717, 444)), ((2, 0, 2), 12, [2048], (38.0, 40.0, 46.1)), ((2, 0, 2), 48, [64], (58.4, 66.5, 64.7)), ((2, 0, 2), 48, [70] + [1] * 15, (162, 173, 173)),
    ((2, 0, 2), 128, [2048], (623, 682, 433)), ((2, 0, 2), 64, [600] * 8, (343, 346, 261)), ((2, 1, 2), 16, [1024] + [1] * 15, (142, None, 155)),
    ((2, 1, 2), 128, [200], (125, None, 101)), ((2, 1, 2), 128, [257], (183, None, 177)), ((2, 1, 2), 128, [2048], (1473, None, 1178)), ((2, 1, 2), 16, [2048], (59.2, None, 69.8)),
    ((2, 1, 2), 12, [251, 180, 60, 30, 12, 6, 4], (75.2, None, 111.8)), ((2, 1, 2), 64, [100, 300, 500, 700, 900], (246, None, 183)), ((2, 1, 2), 64, [2048] + [1] * 20, (824, None, 647))]


@pytest.mark.parametrize("widths,heads,rows,us", STEPS)
def test_no_step_is_slower_than_in_the_one_tile_kernel(widths, heads, rows, us):
    if not native.available():
        pytest.skip("native library not built")
    choice = us[native.lib().cuteafd_latent_prefill_tiles(*widths, heads, len(rows), sum(rows), max(rows))]
    assert choice is not None and choice <= 1.04 * us[0]
    if us[2] < 0.8 * us[0]:
        assert choice == us[2]
