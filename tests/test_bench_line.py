"""The benchmark's printed line stays short whatever its SCF runs carry, and keeps
the keys that its readers take."""
import json


def test_printed_line():
    import bench
    scf = {"workload": "w" * 600, "converged": {"mixed": True, "fp64": True},
           "iterations": {"mixed": 204, "fp64": 216},
           "time_to_eps_s": {"mixed": 83.88, "fp64": 301.75},
           "free_energy_ha": {"mixed": -2339.712572712345, "fp64": -2339.712793271234},
           "free_energy_diff_ha_per_atom": 4.307765432101e-07,
           "last_step_change_ha_per_atom": {"mixed": 1.9e-08, "fp64": 1.9e-08},
           "free_energy_mixed": [-2339.71257271] * 300, "free_energy_fp64": [-2339.71] * 300,
           "diff_charge_fp64": [1e-6] * 300}
    out = {"metric": "m" * 72, "value": 2264.0, "unit": "GB/s", "n_gpus": 1, "steps": 20,
           "warmup": 5, "ms_per_step": 8.174, "higher_is_better": True, "scaling": "weak",
           "vs_baseline": None, "dtype": "f32", "data": "d" * 70,
           "config": {"workload": "w" * 100, "grid": [128] * 3, "bands": 1100, "atoms": 512,
                      "projectors": 12, "inverse_entries": 638784, "l2": "l" * 45,
                      "stencil_staging": "tma", "parallelism": "p" * 30},
           "band_points_per_s": 282250000000.0,
           "roofline": {"bound": "hbm", "kernel": "k_stencil_f32_tma", "achieved": 4700.1,
                        "peak": 6536.4, "unit": "GB/s", "frac": 0.7191, "traffic": 19000000000,
                        "traffic_source": "t" * 120, "ms_per_launch": 3.9},
           "roofline_sweep": {"kernels": "k" * 60, "achieved": 2400.0, "frac": 0.36},
           "e2e": {"value": 99.9, "unit": "GB/s", "h2d_bytes_per_step": 9227468800,
                   "d2h_bytes_per_step": 9227468800, "bands": 1100,
                   "entry_point": "rs_hpsi_host_f32", "equals_device_sweep": True},
           "gpu_launches": 60,
           "clocks": {"sm_mhz": 1965, "sm_max_mhz": 1965, "reasons": ["sw_power_cap"],
                      "samples": 800, "source": "nvml"},
           "cpu_baseline": {"value": 2.213, "unit": "GB/s", "cores": 16, "kind": "port",
                            "sample": "s" * 120, "band_points_per_s": 146297084.6},
           "parity": {"bands": 16, "against": "a" * 110, "nl_dot_f64_bitexact": True,
                      "hpsi_f64_bitexact": True, "max_abs_err_f64": 0.0,
                      "max_rel_err_f32": 1.234567890123e-06},
           "fp64_sweep": {"ms_per_step": 30.1, "gbs": 1200.0, "band_points_per_s": 1e11},
           "scf": scf, "scf_si64": scf}
    line = bench.printed(out)
    assert len(json.dumps(line)) < 2900
    assert line["scf"]["time_to_eps_s"] == scf["time_to_eps_s"]
    for k in ("value", "e2e", "gpu_launches", "ms_per_step", "scaling", "vs_baseline"):
        assert line[k] == out[k]
    assert line["config"]["workload"] == out["config"]["workload"]
    assert line["clocks"]["reasons"] == ["sw_power_cap"]
