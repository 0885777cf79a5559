"""The byte model of the fused stage kernel and the traffic measured against it (no GPU): what
bench.py's roofline of every form is made of, at the 3,145,728-tet channel."""
import pytest

import bench
from test_bench_host import F, N, NB, NODES


@pytest.mark.parametrize("precision,mb", [("fp64", 804.1), ("mixed", 795.4), ("mixed32", 667.9)])
def test_stage_bytes_per_launch(precision, mb):
    assert round(bench.stage_bytes(N, NB, NODES, precision, True) / 1e6, 1) == mb


def test_separate_kernels_of_the_fp32_copies():
    alg = bench.algorithmic_bytes(N, F, NB, NODES, "mixed32", True)
    assert round(alg["gradient"] / 1e6, 1) == 463.3 and round(alg["flux"] / 1e6, 1) == 866.0


def test_every_benched_form_has_measured_traffic():
    assert set(bench.STAGE_DRAM_BYTES_PER_CELL) == {"fp64", "mixed"}
    assert set(bench.MEASURED_DRAM_BYTES_PER_CELL) == {("mixed32", "gradient"), ("mixed32", "flux")}
    for precision, per_cell in bench.STAGE_DRAM_BYTES_PER_CELL.items():
        assert 0.9 <= per_cell * N / bench.stage_bytes(N, NB, NODES, precision, True) <= 1.1, precision
