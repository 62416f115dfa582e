"""How calls are cut up for the device, by size: host arithmetic, no GPU."""
import pytest

SMS = 148


def _tiles(out, rows):
    return -(-out // 128) * -(-rows // 256)


# q / k / v and gate / up of hidden sizes that a decoder has: with few rows all of a group's CTAs run side by side.  (More than the SMs cost
# 20 to 35 %.)
GROUPS = [(1024, (1024, 256, 256), 1024), (1024, (1024, 1024, 1024), 512), (1024, (4096, 4096), 256), (1280, (1280, 256, 256), 1024),
          (1536, (1536, 1536, 1536), 256), (1792, (1792, 256, 256), 512), (2048, (2048, 256, 256), 256), (2048, (2048, 512, 512), 256),
          (2048, (2048, 2048), 256), (2048, (3072, 768, 768), 256), (2560, (2560, 512, 512), 256), (3072, (1024, 1024, 1024), 256)]


@pytest.mark.parametrize("cols,outs,most", GROUPS)
def test_groups_fit_the_device(cols, outs, most):
    from turboquant_mlx_core_b200 import _lib
    lib = _lib.load()
    for rows in (9, 16, 32, 64, 128, 256, 300, 512, 1024):
        if rows <= most:
            assert sum(_tiles(o, rows) * lib.tq_linear_k_splits(o, cols, rows, 1, SMS) for o in outs) <= SMS, rows


def test_splits_of_k():
    """Eight blocks of 64 columns a split at least, no more CTAs than SMs, at least one split."""
    from turboquant_mlx_core_b200 import _lib
    lib = _lib.load()
    for planes in (1, 2):
        for cols in (64, 512, 768, 960, 1024, 1088, 4096, 18944, 28672):
            for out in (1, 512, 3584, 8192, 37888, 151936):
                for rows in (9, 256, 257, 2048):
                    s = lib.tq_linear_k_splits(out, cols, rows, planes, SMS)
                    assert s >= 1 and (s == 1 or (cols // 64 * planes // s >= 8 and s * _tiles(out, rows) <= SMS))
    assert lib.tq_linear_k_splits(8192, 512, 128, 1, SMS) == 1     # (the sums would outweigh what the CTAs gain)
    assert lib.tq_linear_k_splits(512, 100, 9, 1, SMS) == -1 and lib.tq_linear_k_splits(512, 128, 0, 1, SMS) == -1
