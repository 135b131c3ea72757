"""The bench line's summary of the Q2 workload reports the calls a caller gets by default, not the tensor-core contraction
that has to be asked for."""
import bench


def test_q2_summary_is_of_the_default_path():
    c3 = {"jac_fp32_plus_res_ms": 0.93, "jac_fp32_plus_res_ms_tensor_cores": 1.18, "jac_only_ms": 0.71,
          "jac_only_ms_tensor_cores": 0.84, "roofline": {"hbm_frac": 0.11},
          "roofline_tensor_cores": {"hbm_frac": 0.09, "tensor_frac_issued": 0.3}}
    t = bench.targets_summary({"ms_per_step": 1.0, "c3": c3})["c3"]
    assert (t["jac_fp32_plus_res_ms"], t["jac_only_ms"], t["hbm_frac"], t["tensor_frac_issued"]) == (0.93, 0.71, 0.11, 0.3)
