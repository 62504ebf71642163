"""The inner solve's passes on tiles of widths that are no power of two (9, 13, 17 and 25 vectors): as many
rows as a tile holds and one more, rows split evenly, wraps across tiles, a last vector that is partly
padding.  As tests/test_gpu_cg_tiles.py."""
import pytest

import test_gpu_cg_tiles as tiles

pytestmark = pytest.mark.gpu

SIZES = [((100, 10, 3), (1, 1, 0)), ((99, 11, 2), (1, 1, 1)), ((52, 19, 4), (0, 1, 0)), ((49, 20, 3), (1, 1, 0)),
         ((133, 16, 2), (1, 0, 0)), ((36, 29, 5), (1, 1, 1)), ((50, 10, 3), (1, 1, 0)), ((17, 29, 2), (1, 1, 0))]


@pytest.mark.parametrize("precision,tol,bound", [("fp64", 1e-13, 1e-10), ("mixed", 1e-10, 1e-9)])
@pytest.mark.parametrize("dims,periodic", SIZES)
def test_tile_widths(cuda_lib, dims, periodic, precision, tol, bound):
    tiles.test_tile_edges(cuda_lib, dims, periodic, precision, tol, bound)
