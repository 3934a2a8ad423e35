"""The bench line cites ncu figures only beside the kernel shape that they were
taken on."""
import bench


def test_figures_of_another_shape_are_not_cited():
    tr = bench.traffic_from_profiles()
    taken = tr["capture"]["variants"]
    for kernel in ("list_mixed_cell", "list_mixed_part"):
        for v in taken[kernel]:
            got = bench.captured(tr, kernel, v)
            assert got["bytes"] > 0 and 0 < got["fma_pipe_pct"] < 100 and got["note"]
        assert not set(taken[kernel]) & {8, 10, 14}
        for v in (8, 10, 14):
            assert bench.captured(tr, kernel, v) == {}
        assert bench.captured({}, kernel, taken[kernel][0]) == {}
