"""HYC_TILE's shape holds for every launch: the tile kernel of that shape runs
at sizes that a free launch gives to the strip kernels."""
import pytest

import dispatch


@pytest.mark.parametrize("shape,tma", [("32x16", {0: "tma", 1: "tma", 2: "tma", 4: "tma"}),
                                       ("16x16", {0: "tma", 1: "tma", 2: "tma", 4: "tma"}),
                                       ("32x32", {0: "plain", 1: "plain", 2: "tma", 4: "tma"})])
def test_fixed_shape(built_lib, tmp_path, shape, tma):
    exe = dispatch.build(tmp_path)
    big = [(s, 4500, 3298, 41, 2) for s in (0, 1, 2, 4)]
    assert dispatch.routes(exe, big, shape) == [f"tile {shape} {tma[s]}" for s in (0, 1, 2, 4)]
    assert dispatch.routes(exe, big) == ["strip"] * 4
