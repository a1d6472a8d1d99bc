"""The CPU checks of the packed sweep's window words, activity masks and row maxima for the
shapes that only the default pick uses."""
import pytest

import test_activity_mask as masks
import test_row_argmax as argmax
import test_window_words as words

SHAPES = [(1, 17), (32, 2), (32, 5), (8, 17), (16, 17)]


@pytest.mark.parametrize("g,k", SHAPES)
def test_words_masks_and_row_maxima(g, k):
    words.test_window_bytes_and_load_bounds(g, k)
    masks.test_masks_mark_the_cells_inside_the_row(g, k)
    argmax.test_row_max_and_first_cell(g, k)
