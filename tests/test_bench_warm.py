"""The benchmark's warm-up (bench.warm_up) against the library's rule for graphs: the timed steps replay graphs that
exist, from the state the contract asks for."""
import ctypes as C
import os
import re

import pytest

import bench

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


class _Fake:
    """ecg_api.cu's advance: direct steps first, then captured pairs by the state buffer they start from."""

    def __init__(self):
        self.direct, self.cur, self.graphs, self.since_upload = 0, 0, set(), None
        self.dt, self.t, self.iteration = C.c_double(1e-15), C.c_double(0.), 0

    def upload(self, fields):
        self.fields, self.since_upload = fields, 0

    def step(self, n):
        self.since_upload += n
        self.iteration += n
        if n:
            self.dt.value, self.t.value = 1., self.t.value + n
        launched = captured = 0
        while n and self.direct < bench.GRAPH_AFTER:
            self.direct, self.cur, n, launched = self.direct + 1, 1 - self.cur, n - 1, launched + 1
        if n >= 2 and self.cur not in self.graphs:
            self.graphs.add(self.cur)
            captured = 1
        if n % 2:
            self.cur, launched = 1 - self.cur, launched + 1
        return launched, captured


@pytest.mark.parametrize("warmup", [0, 3, 4, 5, 50])
def test_timed_steps_replay_existing_graphs(warmup):
    ctx = _Fake()
    bench.warm_up(ctx, "fields", warmup)
    assert ctx.since_upload == warmup and ctx.iteration == warmup and ctx.t.value == warmup
    assert (warmup == 0) == (ctx.dt.value == 1e-15)
    assert ctx.step(200) == (0, 0)


def test_graph_rule_is_the_librarys():
    src = open(os.path.join(ROOT, "ecogen_b200", "csrc", "ecg_api.cu")).read()
    assert int(re.search(r"#define ECG_GRAPH_AFTER (\d+)", src).group(1)) == bench.GRAPH_AFTER
