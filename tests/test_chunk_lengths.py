"""The kernels that march down chunks of levels, with chunks as long as large grids give them.

cgrd_levels (split step) cuts a column into as many chunks as give the device about 128 warps an SM, of at
least four levels; march_grid (FP64 step) takes two to eight levels.  A warp is 32 rows, so few rows and many
columns give the warps of a large grid with a fraction of its cells: here chunks of 17 in two and of a whole column
of 21 levels (split), and of eight (FP64), with flat and terrain-following layers in one chunk.  The checks are
those of the small grids: every marching kernel's fields against the FP64 step, the state against it, and
the FP64 step against the oracle.
"""
import pytest

import lgame_gpu as L
from test_column_tiles import test_split_close_to_fp64_at_the_tilings_borders as state_close_to_fp64
from test_fp64_columns import test_fp64_columns_match_oracle as fp64_matches_oracle
from test_marching_kernels import test_marching_kernels_close_to_fp64 as fields_close_to_fp64

SMS = 152


def split_chunk(ny, nx, nl):
    """levels a chunk, as cgrd_levels has it"""
    warps = 4 * ((ny + 31) // 32) * ((nx + 3) // 4)
    chunks = min(-(-SMS * 128 // warps), nl)
    return max(-(-nl // chunks), 4)


def fp64_chunk(ny, nx, nl):
    """levels a chunk, as march_grid has it"""
    return min(8, max(2, 128 * ((ny + 31) // 32) * ((nx + 3) // 4) * nl // (SMS * 1536)))


# (ny, nx, n_layers, n_oro_layers), levels a chunk
SPLIT = [((3, 9729, 34, 25), 17), ((3, 19457, 21, 16), 21)]


@pytest.mark.gpu
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("grid, length", SPLIT)
def test_split_marching_kernels_in_long_chunks(grid, length, periodic):
    ny, nx, nl, _ = grid
    assert split_chunk(ny, nx, nl) == split_chunk(ny + 1, nx + 1, nl) == length
    fields_close_to_fp64(grid, periodic)


@pytest.mark.gpu
@pytest.mark.parametrize("grid, length", SPLIT)
def test_split_state_in_long_chunks(grid, length):
    state_close_to_fp64(grid, L.PRECISION_SPLIT)


@pytest.mark.gpu
@pytest.mark.parametrize("periodic", [True, False])
def test_fp64_step_in_long_chunks(periodic):
    ny, nx, nl, no = 3, 1501, 41, 30
    assert fp64_chunk(ny, nx, nl) == 8
    fp64_matches_oracle((ny, nx, nl, no, periodic))
