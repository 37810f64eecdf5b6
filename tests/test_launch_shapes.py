"""The launch-shape rules around the tuned table (CPU): second rounds, uneven
batches and the shortest signal's share, over a table written here and over
the committed ones."""
import math

import pytest

from eemd4cuda_b200 import autotune as A

TABLE = [(8192, 32, 16, 4), (8192, 64, 8, 4), (49152, 64, 6, 4), (49152, 100, 4, 5), (49152, 1024, 1, 4)]


@pytest.fixture
def table(monkeypatch):
    monkeypatch.setattr(A, "_table", lambda dtype: TABLE)
    A._SHAPES.clear()
    yield
    A._SHAPES.clear()


def test_no_second_round_for_a_few_more_tasks(table):
    # 6 CTAs per task: 98 tasks at once in float32 (592 slots), 74 in float64 (444)
    assert A.launch_shape(49152, 70, "f64") == (6, 4)
    assert A.launch_shape(49152, 75, "f64") == (4, 5)
    assert A.launch_shape(49152, 80, "f32") == (6, 4)


def test_longest_signal_bounds_the_tail(table):
    even = A.launch_shape(49152, 960, "f32")
    assert even == (1, 4)
    lengths, trials = [4096, 49152, 262144], 320
    total = sum(lengths) * trials
    c, w = A.launch_shape(49152, 960, "f32", n_min=4096, n_max=262144, total=total)
    slots = A.SMS * 4
    assert (c, w) == (min(16, max(1, math.ceil(262144 * slots / (1.5 * total)))), 4)
    # a median-sized longest signal asks for nothing more
    assert A.launch_shape(49152, 960, "f32", n_min=4096, n_max=60000, total=total) == even


@pytest.mark.parametrize("n_min,c", [(8192, 16), (8191, 15), (1024, 2), (1023, 1), (5, 1)])
def test_shortest_signal_keeps_the_entrys_share(table, n_min, c):
    # the 8192 entry was measured with 512 samples per CTA, so that is its floor
    assert A.launch_shape(8192, 32, "f64", n_min=n_min) == (c, 4)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_committed_tables_give_launchable_shapes(dtype):
    for n in (1, 3, 513, 2048, 3001, 8192, 48000, 300000, 1 << 22):
        for tasks in (1, 7, 75, 1000, 100000):
            for n_max in (n, 5 * n):
                c, w = A.launch_shape(n, tasks, dtype, n_min=max(1, n // 3), n_max=n_max, total=n * tasks + 4 * n)
                assert 1 <= c <= 16 and w in A.WARPS
                assert c == 1 or max(1, n // 3) // c >= A.GRAIN
