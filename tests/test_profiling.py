"""Figures of an ncu capture: launches of a pass added up, passes averaged."""
import pytest

from rkhs_ba_gb300 import profiling

RAW = '''"ID","Kernel Name","dram__bytes_read.sum","dram__bytes_write.sum","smsp__inst_executed.sum","gpu__time_duration.sum"
"","","Mbyte","Kbyte","inst","us"
"0","void k_rows<2, 0, 0, 1, 0>(BatchDev)","40","500","1,000","600"
"1","void k_cand<2>(BatchDev)","10","100","200","100"
"2","void k_rows<2, 0, 0, 1, 1>(BatchDev)","20","0","300","50"
"3","void k_gradient(BatchDev)","999","999","999","999"
"4","void k_rows<2, 0, 0, 1, 0>(BatchDev)","42","500","1,200","620"
"5","void k_cand<2>(BatchDev)","10","100","200","100"
"6","void k_rows<2, 0, 0, 1, 1>(BatchDev)","22","0","100","30"
'''


def test_pass_of_several_kernels():
    m = profiling.read_raw(RAW, "k_cand,k_rows", 3)
    assert m == {"dram__bytes_read.sum": 72e6, "dram__bytes_write.sum": 0.6e6, "smsp__inst_executed.sum": 1500.0,
                 "gpu__time_duration.sum": 750e3}


def test_single_kernel_is_averaged():
    assert profiling.read_raw(RAW, "k_cand")["smsp__inst_executed.sum"] == 200.0


def test_incomplete_pass_is_refused():
    with pytest.raises(ValueError):
        profiling.read_raw(RAW, "k_cand,k_rows", 4)


def test_committed_summary_has_what_the_bench_reads():
    d = profiling.load("k_rows_global50k.json")
    assert d["launches_per_pass"] == 3 and d["dram_bytes_per_pair_launch"] > 0 and d["warp_instructions_per_pair_launch"] > 0
