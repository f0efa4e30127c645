"""The roofline line of bench.py names the SpMV kernel that ran and takes that
kernel's DRAM traffic (CPU only)."""
import os

import bench

LINE = "parrsb_gb300: SpMV autotune tiles=%d groups=4 rows=8388608 -> %s x 512\n"


def test_kernels_of_the_log():
    log = LINE % (1024, "k_spmv_loc") + "other output\n" + LINE % (2048, "k_spmv")
    assert bench.spmv_kernels(log) == ["k_spmv", "k_spmv_loc"]
    assert bench.spmv_kernels("") == []


def test_traffic_belongs_to_the_kernel():
    loc, plain = bench.load_traffic(["k_spmv_loc"]), bench.load_traffic(["k_spmv"])
    assert loc["source"] != plain["source"]
    assert loc["dram_bytes_per_algorithmic_byte"] != plain["dram_bytes_per_algorithmic_byte"]
    for kernels in ([], ["k_spmv", "k_spmv_loc"], ["k_spmv_tma"]):
        assert bench.load_traffic(kernels) is None


def test_capture(capfd):
    with bench.StderrCapture() as log:
        os.write(2, b"from the library\n")
    assert log.text == "from the library\n"
    assert "from the library" in capfd.readouterr().err
