"""What bench.py says of a build whose box, keys and sort are one kernel (CPU only)."""
import bench

STAGES = {"bounds": 0.006, "morton": 0.002, "sort": 0.021, "gather": 0.0, "tree": 0.008, "top": 0.010}


def test_a_small_build_reports_the_kernels_it_launches():
    n = bench.SMALL_BUILD
    name, ms, nbytes, traffic = bench.dominant_kernel(STAGES, n)
    assert name == "k_small_sort" and abs(ms - 0.029) < 1e-12 and nbytes == 56 * n
    assert traffic is None  # no capture of it is kept
    slow_tree = dict(STAGES, tree=0.1)
    assert bench.dominant_kernel(slow_tree, n)[:2] == ("k_tree_climb", 0.1)
    assert bench.launches_per_build(n) == 3 and bench.launches_per_build(n + 1) == bench.LAUNCHES_PER_BUILD


def test_a_large_build_is_reported_as_before():
    n = 1 << 24
    stages = {"bounds": 0.17, "morton": 0.08, "sort": 0.4, "gather": 0.0, "tree": 0.8, "top": 0.07}
    name, ms, nbytes, traffic = bench.dominant_kernel(stages, n)
    assert name == "k_tree_climb" and ms == 0.8 and nbytes == bench.MODEL_BYTES["tree"] * n
    assert traffic == bench.load_traffic("k_tree_climb", n)
    name, ms, nbytes, _ = bench.dominant_kernel(dict(stages, sort=3.0), n)
    assert name == "k_scatter" and ms == 1.0 and nbytes == bench.MODEL_BYTES["sort"] * n / 3


def test_the_note_on_l2_follows_the_size():
    assert bench.l2_note(1 << 24) == "input soup 805 MB > 126 MB L2; no flush"
    assert "fits" in bench.l2_note(65_536)


def test_the_line_says_whether_a_graph_runs():
    with open(bench.__file__) as f:
        src = f.read()
    assert '"graph": n > SMALL_BUILD' in src and '"graph": True' not in src
