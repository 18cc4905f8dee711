"""The benchmark's printed line holds the contract's keys and stays short enough
to be read whole from the end of the output, whatever the modes measured."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

CONTRACT = {"metric": "frames/s", "value": 3712.123456789, "unit": "frames/s", "n_gpus": 1, "steps": 512, "warmup": 5,
            "ms_per_step": 0.26938712345, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": "synthetic", "gpu_launches": 3584}


def test_line_is_short_and_complete():
    import bench
    rate = {"rate_req_s": 200, "frames_per_s": 201.8009991162081, "p99_ms": 62.767041919998874}
    line = dict(CONTRACT, config=bench.workload_config(bench.CONFIGS["plain2048"], 1),
                e2e={"value": 3342.9253003301665, "unit": "frames/s", "h2d_bytes_per_step": 919987,
                     "d2h_bytes_per_step": 8294400, "note": "n" * 200},
                roofline={"bound": "hbm", "achieved": 1852.876418293033, "peak": 6787.2, "unit": "GB/s",
                          "frac": 0.2729957004792894, "traffic": None, "traffic_note": "t" * 300,
                          "algorithmic_bytes_per_launch": 411762498.4, "kernel": "raycast_tiles_kernel<u8,trilinear>",
                          "peak_source": "MEASURED_PEAKS.json hbm_gbs"},
                clocks={"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []},
                cpu_baseline={"value": 3.6275, "unit": "frames/s", "cores": 16, "cpu_model": "Neoverse-V2", "kind": "port",
                              "lod_select_ms": 1.25, "sample": "s" * 160},
                served=dict({k: rate for k in ("capacity_served", "capacity_plain")}, rates=[rate] * 40,
                            rate_at_p99_slo=[rate] * 6),
                batched=dict({k: dict(rate, config={"tile_w": 8}) for k in ("plain", "batched", "persistent")},
                             autotune_table=[["x", 8, 8, 0.123456789]] * 44, speedup_frames_per_s=1.0761520838449337),
                parity={"tolerance": 1 / 255, "plain256": [{"rows": "all"}] * 50, "max_err_255": 0.0127217053672668},
                plain256={"workload": "w", "frames_per_s": 7302.014931897775},
                outofcore={"workload": "w", "frames_per_s": 15.332745555228952, "generator": "g" * 200},
                launch_sweep_raycast_ms={"tile grid %d" % i: 0.2391234567 for i in range(20)})
    for k in ("p50_ms", "p99_ms", "samples_per_s", "raycast_ms_mean", "select_ms_mean", "wall_s", "volume_generation_s"):
        line[k] = 0.123456789012
    text = json.dumps(bench.compact(line))
    assert len(text) < 3000
    out = json.loads(text)
    assert {k: out[k] for k in CONTRACT} == CONTRACT
    assert out["config"] == line["config"] and out["clocks"] == line["clocks"]
    assert {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"} <= set(out["e2e"])
    assert out["batched"]["batched"] == 201.801 and out["served"]["capacity_served"]["rate_req_s"] == 200
