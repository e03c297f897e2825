"""The counters that bench.py combines with its own times (profiles/ncu_metrics.json):
a record of the step kernel for each mode of the headline workload."""
import bench


def test_a_record_for_each_mode():
    for key in ("lean_step_kernel_euler1280x320", "lean_step_kernel_split_euler1280x320"):
        rec = bench._ncu_record(key)
        assert rec is not None, key
        assert rec["cells"] == 1280 * 320
        # a state of 13.1 MB is read, and a cell's FP64 operations are between one and two thousand
        # unsplit, fewer split
        assert rec["dram_bytes_read"] > 13e6 and rec["dram_bytes_write"] >= 0
        per_cell = 32 * rec["fp64_pipe_warp_inst"] / rec["cells"]
        assert rec["fp64_pipe_warp_inst"] < rec["warp_inst"] and 500 < per_cell < 2000, per_cell
