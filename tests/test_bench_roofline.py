"""The benchmark line names the sweep kernel that ran and what bounds it: one
launch per colour, passes of two iterations, or the resident sweeps of grids up
to 128^3, which run hundreds of iterations a launch."""
import pytest

from test_bench_contract import load_bench


@pytest.mark.parametrize("n, sweeps, launches, kernel, bound, bytes_per_cell", [
    (128, 5000, 10000, "k_sor_rbz", "hbm", 6.0),
    (256, 5696, 2848, "k_sor_wave", "hbm", 12.0),
    (256, 236, 117, "k_sor_wave", "hbm", 12.0),  # the count of a CG solve's applications is rounded
    (128, 2600, 5, "k_sor_resident", "latency", 12.0),
    (64, 8, 1, "k_sor_resident", "latency", 12.0),
])
def test_sweep_kernel_by_the_form_that_ran(n, sweeps, launches, kernel, bound, bytes_per_cell):
    line = load_bench().sweep_roofline({"sor": {"ms": 10.0, "launches": launches}}, sweeps, n ** 3, 6000.0, "measured")
    assert line["kernel"].split()[0] == kernel and line["bound"] == bound
    assert line["bytes_per_launch"] == bytes_per_cell * n ** 3
    assert line["half_sweep_us"] == pytest.approx(10e3 / (2 * sweeps))
    assert line["achieved"] == pytest.approx(line["bytes_per_launch"] * launches / 10e-3 / 1e9)
