"""The cases of the GPU tests reach every fp32 kernel that they are there for: the rules that choose one, no GPU."""
from test_gpu_parity import FEW_ROWS, FEW_ROWS_NETS, FFMA_WINDOWS
from test_gpu_tcgemm import CHAIN_K, CHAIN_SHAPES

PLAIN, FORWARD, ERRPROP, GRAD = range(4)
FEW_NODES, BY_ROWS, TILES = range(3)


def test_few_rows_reach_every_product_by_rows(g):
    for sizes in FEW_ROWS_NETS[2:]:
        for rows in FEW_ROWS:
            routes = [g.ffma_route(FORWARD, rows, sizes[l + 1], sizes[l]) for l in range(len(sizes) - 1)]
            if rows <= 32:
                block = next(b for b in (1, 8, 16, 32) if rows <= b)
                assert routes == [(BY_ROWS, block)] * len(routes), (sizes, rows)
            else:
                assert all(r[0] == TILES for r in routes) or rows >= 64, (sizes, rows)
    for sizes in FEW_ROWS_NETS:
        assert all(g.ffma_route(FORWARD, 700, sizes[l + 1], sizes[l])[0] != BY_ROWS for l in range(len(sizes) - 1))


def test_windows_reach_every_tile_of_every_product(g):
    seen = set()
    for sizes, rows, mom, _ in FFMA_WINDOWS:
        for l in range(len(sizes) - 1):
            ni, no = sizes[l], sizes[l + 1]
            seen.add((FORWARD, False) + g.ffma_route(FORWARD, rows, no, ni))
            seen.add((GRAD, mom > 0) + g.ffma_route(GRAD, no, ni, rows))
            if l >= 1:
                seen.add((ERRPROP, False) + g.ffma_route(ERRPROP, rows, ni, no))
    for kind in ((FORWARD, False), (ERRPROP, False), (GRAD, False), (GRAD, True)):
        for tile in (32, 64, 96, 128):
            assert kind + (TILES, tile) in seen, (kind, tile)
        assert kind[0] == ERRPROP or kind + (FEW_NODES, 0) in seen, kind


def test_plain_products_turn_the_ring_on_every_tile(g):
    seen = {g.ffma_route(PLAIN, M, N, K) for M, N, _ in CHAIN_SHAPES for K in CHAIN_K if K > 4 * 32}
    assert {(TILES, t) for t in (32, 64, 96, 128)} <= seen
    # the 32 rows that each of them is compared with
    assert all(g.ffma_route(PLAIN, 32, N, K) == (TILES, 32) for _, N, _ in CHAIN_SHAPES for K in CHAIN_K)
