"""The order in which the tensor-core kernels' CTAs take the items of an exact causal launch (csrc/attn_items.cuh), worked out on the host by the
kernels' own functions."""
import ctypes as C
import os
import subprocess
import sys

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'hyperattention_b200', 'csrc')
SOURCE = r'''
#include "attn_items.cuh"
using namespace ha;
// places and segments of the items in the order of turns (places[turn * grid + cta]; -1: none); returns the number of turns
extern "C" int deal(int places, int segs, int rows, int d, int width, int sms, int* place, int* seg, int* meta) {
  ha_attn_params p{};
  p.mode = HA_MODE_FLASH; p.flags = HA_FLAG_CAUSAL; p.dtype = HA_BF16;
  p.B = 1; p.H = segs; p.n = p.m_q = p.m_k = rows; p.span = rows; p.segs_per_head = 1; p.d = p.dv = d;
  AttnPlan pl;
  pl.pairs = places; pl.n_items = segs * places; pl.by_pairs = FastDiv(places);
  const int grid = pl.n_items < sms ? pl.n_items : sms;
  plan_order(pl, p, grid, width);
  const int turns = (pl.n_items + grid - 1) / grid;
  for (int t = 0; t < turns; ++t)
    for (int c = 0; c < grid; ++c) {
      const int item = item_of_turn<true>(pl, t, c, grid);
      place[t * grid + c] = -1;
      if (item < pl.n_items) place[t * grid + c] = causal_place(pl, item, seg[t * grid + c]);
    }
  meta[0] = grid; meta[1] = pl.by_length; meta[2] = pl.by_length ? pl.round_segs : 0; meta[3] = pl.by_length ? pl.rest_segs : 0;
  meta[4] = pl.by_length ? pl.whole_segs : 0;
  return turns;
}
'''
SMS = 148


@pytest.fixture(scope='module')
def deal(tmp_path_factory):
    sys.path.insert(0, CSRC)
    import build
    src = tmp_path_factory.mktemp('order') / 'order.cu'
    src.write_text(SOURCE)
    lib = str(src)[:-3] + '.so'
    subprocess.run([os.environ.get('NVCC', 'nvcc')] + build.NVCC_FLAGS + ['-shared', str(src), '-o', lib], check=True, timeout=300)
    lib = C.CDLL(lib)

    def run(places, segs, rows, d, width=2):
        n = segs * places + SMS
        place, seg, meta = (C.c_int * n)(), (C.c_int * n)(), (C.c_int * 5)()
        turns = lib.deal(places, segs, rows, d, width, SMS, place, seg, meta)
        grid = meta[0]
        ctas = [[(place[t * grid + c], seg[t * grid + c]) for t in range(turns) if place[t * grid + c] >= 0] for c in range(grid)]
        return ctas, meta
    return run


def longest(ctas, places):
    """key tiles of the longest CTA over the average of all SMs (an item of place p: 2 (places - p) of them, and one for its start)"""
    loads = [sum(2 * (places - p) + 1 for p, _ in items) for items in ctas]
    return max(loads) / (sum(loads) / SMS)


@pytest.mark.parametrize('d', [64, 128])
@pytest.mark.parametrize('places', [1, 2, 3, 4, 5, 7, 8, 9, 13, 16, 22, 32, 33, 64])
def test_every_item_is_taken_once(deal, places, d):
    for segs in (1, 2, 5, 18, 32, 37, 74, 104, 148, 149, 230, 295, 296, 297, 400, 513):
        ctas, _ = deal(places, segs, 256 * places, d, 4 if segs % 2 else 2)
        items = [x for items in ctas for x in items]
        assert sorted(items) == [(p, s) for p in range(places) for s in range(segs)], (places, segs)


@pytest.mark.parametrize('places,segs,bound', [(3, 400, 1.12), (5, 400, 1.08), (5, 512, 1.08), (7, 400, 1.07), (8, 400, 1.07), (14, 320, 1.11), (16, 320, 1.04),
                                               (19, 320, 1.05), (22, 320, 1.07), (23, 320, 1.06), (31, 320, 1.04)])
def test_own_order_is_turned_so_that_a_cta_meets_all_lengths(deal, places, segs, bound):
    """launches that keep the segments' own order (more than two segments a CTA): the longest CTA stays near the average"""
    ctas, meta = deal(places, segs, 256 * places, 128)
    assert not meta[1]
    assert longest(ctas, places) < bound


@pytest.mark.parametrize('places,segs,rows,d,width', [(8, 64, 2048, 128, 2), (8, 72, 2048, 128, 2), (16, 32, 4096, 128, 2), (32, 32, 8192, 64, 2), (12, 104, 3072, 64, 2),
                                                      (16, 38, 2048, 128, 4), (24, 85, 3072, 128, 4), (24, 85, 6144, 64, 4)])
def test_few_segments_are_dealt_out_by_length(deal, places, segs, rows, d, width):
    """launches of a few segments a CTA whose shared rows fit L2: hardly a CTA has more than its part"""
    ctas, meta = deal(places, segs, rows, d, width)
    assert meta[1] and longest(ctas, places) < 1.06


@pytest.mark.parametrize('width', [2, 4])
@pytest.mark.parametrize('d', [64, 128])
def test_what_is_live_at_once_stays_near_l2(deal, d, width):
    """the rounds and what is left after them (up to two turns of the grid more than a round) share no more than 160 MiB of rows"""
    for places in range(1, 49):
        rows = (128 if (d, width) == (128, 4) else 256) * places          # (128 wide backward: an item is a key tile)
        for segs in range(1, 300, 7):
            _, (_, by_length, round_segs, rest_segs, whole_segs) = deal(places, segs, rows, d, width)
            if by_length:
                assert max(round_segs if whole_segs else 0, rest_segs) * rows * 2 * d * width <= 160 << 20, (places, segs)
