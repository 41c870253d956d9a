"""The benchmark's printed line: short enough to come through whole, with every
key that a reader of it needs; the full record goes to standard error."""
import json

import bench


def _record():
    """A full record of the size that a run on all legs makes (20,000 characters)."""
    f, text = 12345.678901234567, "x" * 300
    phases = {p: {f"field_{i}": f for i in range(40)} for p in ("global_relabel", "push", "inside_full_solve")}
    roofline = dict(bound="hbm", kernel="solve", achieved=f, peak=f, unit="GB/s", frac=0.5080377153267878,
                    peak_source="of measured (MEASURED_PEAKS.json hbm_gbs)", traffic=f * 1e6,
                    alg_bytes_per_launch=f * 1e6, avg_launch_us=f, share_of_step=0.61, kernels_ms={"solve": f},
                    solve_phases=phases)
    e2e = dict(value=f, unit="Mpixel/s", h2d_bytes_per_step=187475996, d2h_bytes_per_step=93737998, ms_per_step=f,
               api=text)
    leg = dict(desc=text, images=1, value=f, unit="Mpixel/s", ms_per_step=f, steps=10, e2e=e2e, roofline=roofline)
    tuning = dict(push_rounds_per_gr=2, max_tile_sweeps=16, sweeps_per_local_relabel=4, blocks_per_sm=4, threads_y=8,
                  ms_default=f, ms_best=f, configs_tried=38)
    config = bench.workload_config("batch256", bench.workload("batch256"), 1)
    config.update(tuning=tuning, cuda_graph={"active": True, "captures": 6})
    return dict(metric=bench.METRIC, value=f, unit="Mpixel/s", n_gpus=1, steps=20, warmup=5, ms_per_step=f,
                higher_is_better=True, scaling="weak", vs_baseline=None, dtype="int32",
                data="synthetic (seeded in-repo generator; no dataset)", config=config, e2e=e2e, e2e_sync=e2e,
                roofline=roofline, gpu_launches=100, solver={f"counter_{i}": 10 ** 9 for i in range(24)},
                clocks=dict(sm_mhz=2070.0, sm_max_mhz=2070.0, reasons=["sw_power_cap"], samples=40,
                            window="device-resident and end-to-end timed regions"),
                plain_per_image=dict(e2e, flows_equal_batched=True, cuts_equal_batched=True),
                serving=dict(workload=text, served=dict(p50_ms=f, p99_ms=f, mpixel_s_over_busy=f,
                                                        edit_tail={"slowest": [text] * 6}),
                             p99_target_ms=5.0, p99_met=True, results_equal=True),
                flows_host_equal_device=True, cuts_host_equal_device=True,
                cpu_baseline=dict(value=f, unit="Mpixel/s", cores=1, kind="port", sample="x" * 80),
                parity=dict(images_checked=256, flows_equal_oracle=True, smin_equal_oracle=True,
                            smax_equal_oracle=True),
                reference_cuda=dict(value=f, unit="Mpixel/s", images=12, labels_equal_smax=12, how=text),
                single_image=dict({n: leg for n in (*bench.SINGLE_WORKLOADS, "n8_640x480")},
                                  clocks=dict(sm_mhz=2070.0)))


def test_printed_line_is_short_and_complete(capsys):
    full = _record()
    bench.emit(full)
    out, err = capsys.readouterr()
    assert out.endswith("\n") and out.count("\n") == 1 and len(out) <= 2800
    line = json.loads(out)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "gpu_launches", "clocks", "cpu_baseline", "parity"):
        assert line[k] == full[k]
    assert line["config"]["workload"] == "batch256" and line["config"]["parallelism"] == "shard by image x1"
    assert set(line["e2e"]) >= {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"}
    assert abs(line["e2e"]["value"] / full["e2e"]["value"] - 1) < 1e-6
    assert set(line["roofline"]) >= {"bound", "kernel", "achieved", "peak", "unit", "frac"}
    assert set(line["single_image"]) == {*bench.SINGLE_WORKLOADS, "n8_640x480"}
    assert err.startswith("detail: ") and json.loads(err[len("detail: "):]) == full


def test_a_single_leg_has_a_line_too():
    leg = _record()
    for k in ("e2e_sync", "plain_per_image", "serving", "single_image", "cpu_baseline", "reference_cuda"):
        del leg[k]
    leg["config"] = bench.workload_config("n8_640x480", None, 1)
    line = bench.headline(leg)
    assert line["value"] == leg["value"] and "tuning" not in line["config"]
