"""The forms that prompt rows go through by what the host knows of their batch -- a tile of one slot a CTA, two heads of a kv head or two row tiles a
CTA, CTAs that take tiles in turns -- on both sides of each rule.  Oracle and tolerance are those of test_gpu_prompt_tc5."""
import pytest

from test_gpu_prompt_tc5 import test_gathered_prompt_rows as gathered_rows, test_masked_prompt_rows as masked_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [
    # lens, ctx, heads, kv heads, dk, dv, page, chunk, window, keep, cap, sink, maps, sigmoid, gate, scale factor
    # most sequences are decode rows: counted as more tiles than there are, which turn out to be one wave
    ([1] * 40 + [200, 130], [60] * 40 + [0, 77], 32, 8, 64, 64, 16, 0, 100, 3, 0.0, True, 1, False, True, 1.0),
    ([1] * 40 + [300, 16], [60] * 41 + [5], 28, 4, 64, 64, 16, 0, 0, 0, 0.0, False, 1, False, True, 1.0),
    ([1] * 33 + [250], [60] * 33 + [9], 16, 2, 128, 64, 16, 128, 0, 0, 0.0, False, 1, True, False, 1.0),
    # ... and where capped scores or two maps make the start in turns a long one
    ([1] * 40 + [200], [60] * 40 + [9], 32, 8, 64, 64, 16, 0, 100, 3, 30.0, True, 1, False, True, 1.0),
    ([1] * 40 + [150] + [16] * 9, [60] * 40 + [9] * 10, 32, 8, 64, 64, 16, 0, 100, 3, 0.0, True, 2, False, True, 1.0),
    ([100, 140, 30], [0, 9, 200], 49, 7, 64, 64, 16, 0, 0, 0, 0.0, True, 1, False, False, 1.0),          # two row tiles a CTA of odd heads
    # portions of a few key tiles, two heads a CTA: one wave, the last tile's edges, pages that are no power of two; nine steps, and more than a wave
    ([200, 129, 128, 16, 250, 201, 127, 255], [0, 40, 0, 9, 0, 1, 600, 0], 16, 4, 128, 128, 16, 0, 0, 0, 0.0, True, 1, False, True, 1.0),
    ([290, 411, 130], [0, 33, 5], 32, 8, 64, 64, 24, 300, 100, 7, 0.0, True, 1, False, False, 1.0),
    ([500, 300], [3, 0], 32, 4, 96, 128, 16, 0, 200, 0, 0.0, False, 1, True, False, 1.0),
    ([1020], [30], 32, 8, 64, 64, 16, 0, 0, 0, 0.0, False, 1, False, False, 1.0),
    ([300] * 7, [0] * 7, 16, 4, 64, 64, 16, 0, 0, 0, 0.0, False, 1, False, False, 1.0),
    # capped scores in short windows or blocks: two heads a CTA, scores on both sides of the polynomial; one slot; two row tiles; a longer window
    ([600, 333], [0, 40], 32, 8, 128, 128, 16, 0, 150, 5, 30.0, True, 1, False, True, 1.0),
    ([600, 333], [0, 40], 32, 8, 64, 64, 24, 256, 0, 0, 1.5, False, 1, False, False, 1.0),
    ([400, 500], [5, 0], 28, 4, 64, 64, 16, 0, 200, 0, 30.0, True, 1, False, False, 1.0),
    ([700, 640], [5, 0], 28, 4, 64, 128, 16, 0, 384, 3, 30.0, False, 1, False, True, -1.0),
    ([700, 640], [5, 0], 28, 4, 64, 64, 16, 0, 900, 0, 30.0, False, 1, False, False, 1.0),
])
def test_forms(cuda, c):
    masked_rows(cuda, c)


@pytest.mark.parametrize("lens,ctx,H,dn,dr,dv,window,sink,gate", [
    ([85, 58, 83, 148], [555, 0, 30, 9], 32, 128, 64, 128, 0, True, 1),  # two row tiles a CTA where one a CTA would be more than a wave
    ([1792], [0], 16, 128, 64, 128, 0, True, 2),                         # one causal portion: one slot to 1.6 waves
    ([2400], [0], 16, 64, 64, 64, 0, False, 1),                          # ... two row tiles a CTA, the last one half a slot
    ([2049], [0], 19, 24, 8, 112, 0, True, 0),                           # ... a row in the last tile
    ([2305], [3], 16, 64, 64, 64, 0, False, 1),                          # behind a context: in turns
])
def test_gathered_forms(cuda, lens, ctx, H, dn, dr, dv, window, sink, gate):
    gathered_rows(cuda, lens, ctx, H, dn, dr, dv, window, sink, gate)
