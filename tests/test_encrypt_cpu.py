"""Encryption with binary keys takes two launches: rows of masks, noise and message,
then the product with the key.  By reading the sources: where the second cannot
be added, because its launch fails or a wait in it expires, the bodies it is
missing from are cleared, as they hold messages.  (Neither can be brought about
on a GPU without harm.)  And the loop that clears them, restated, takes exactly
the columns that the loop it follows had not come to."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "idash2019_2_gb300", "csrc")


def _code(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def test_bodies_without_their_product_are_cleared():
    text = _code("key_product.cu")
    launch = re.search(r"cudaError_t launch_key_product\(.*?\n\}\n", text, re.S).group(0)
    assert re.search(r"if \(e != cudaSuccess && !a\.scores\)\s*k_clear_bodies<<<", launch)
    epilogue = text[text.index("kMagicSum"):text.index("tmem_dealloc(tmem")]
    loops = [m.start() for m in re.finditer(r"for \(;[^;]*it < 2 \* my_items; \+\+it\)", epilogue)]
    assert len(loops) == 2 and "uint64_t it = 0;" in epilogue[:loops[0]]
    assert re.search(r"tc_warp_wait\([^;]*\) break;", re.sub(r"\s+", " ", epilogue[loops[0]:loops[1]]))
    assert "!kScores" in epilogue[loops[1]:] and "body[j] = 0;" in epilogue[loops[1]:]


@pytest.mark.parametrize("N", [64, 1024, 2048])
@pytest.mark.parametrize("row_tiles", [1, 3, 40, 200])
def test_every_column_belongs_to_one_warps_part(N, row_tiles, n_coef=None):
    """Tiles, halves and column steps as launch_key_product and the clearing loop
    compute them cover each coefficient of a row once."""
    n_coef, sms, tile_max = n_coef or N, 152, 256
    pad = (n_coef + 15) // 16 * 16
    least = (pad + 2 * tile_max - 1) // (2 * tile_max)
    pairs = min(max(least, (pad + 63) // 64), max(least, sms // row_tiles))
    cols = ((pad + 2 * pairs - 1) // (2 * pairs) + 15) // 16 * 16
    pairs = (pad + 2 * cols - 1) // (2 * cols)
    hit = [0] * N
    for pair in range(pairs):
        for t in range(2):
            n0 = (2 * pair + t) * cols
            w = min(cols, pad - n0) if n0 < pad else 0
            middle = (w // 2 + 15) // 16 * 16
            for half in range(2):
                for lane4 in range(4):
                    for j in range(n0 + (middle if half else 0) + lane4, min(n0 + (w if half else middle), n_coef), 4):
                        hit[j] += 1
    assert hit == [1] * N
