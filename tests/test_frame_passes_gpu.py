"""The start of a renderer's passes (one launch for seeds, path weights,
counters, frame buffer and the tile states of every bounce) and shadow rays
generated before the shading they are added to: frames of several samples at
the largest depth, with one pixel, ragged and several tiles, shadow passes
overlapped or not, graph replays included, against the oracle's CPU frame."""
import pytest

from test_renderer_gpu import run_pair, same_bits, small  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("overlap,graph", [(1, 0), (0, 0), (1, 1)])
@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 3, 8), (17, 3, 40, 1), (33, 29, 3, 8), (16, 16, 2, 0)])
def test_pass_start(wf, orc, dev, small, w, h, spp, depth, overlap, graph):  # noqa: F811
    px, fp, st, o_px, o_fp, o_st = run_pair(wf, orc, dev, small, w, h, frames=2, num_primary_samples=spp,
                                            recursion_depth=depth, shadow_overlap=overlap, use_graph=graph,
                                            sort_path_rays=1, reorder_path_rays=1, morton_kind=2)
    assert st.num_path_rays == o_st.path and st.num_shadow_rays == o_st.shadow
    assert same_bits(fp, o_fp) and same_bits(px, o_px)
