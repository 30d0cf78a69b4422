"""The benchmark's CPU arm prints the one JSON line its callers parse.

`bench.py --impl reference` times the scalar restatement of the reference's arithmetic on the host cores; it
needs no GPU, so its output contract is checked here on a one-second sample.
"""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_reference_arm(*extra):
    cmd = [sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "3",
           "--cpu-seconds", "1", *extra]
    out = subprocess.run(cmd, cwd=ROOT, capture_output=True, text=True, timeout=300, stdin=subprocess.DEVNULL)
    assert out.returncode == 0, out.stderr[-2000:]
    lines = [ln for ln in out.stdout.splitlines() if ln.startswith("{")]
    assert len(lines) == 1, out.stdout
    return json.loads(lines[0])


def test_reference_arm_line_has_the_contract_keys():
    d = run_reference_arm()
    assert d["impl"] == "reference"
    assert d["metric"] == "moe_layer_tokens_per_s" and d["unit"] == "tokens/s"
    assert d["higher_is_better"] is True and d["n_gpus"] == 1 and d["steps"] == 1 and d["warmup"] >= 3
    assert d["value"] > 0 and d["ms_per_step"] > 0
    assert d["config"]["workload"] == "cfg4"              # the default workload of both arms
    assert d["scaling"] == "strong" and d["config"]["tokens_per_step"] == 8192
    assert d["vs_baseline"] is None
    cb = d["cpu_baseline"]
    assert cb["kind"] in ("port", "reference") and cb["cores"] >= 1 and cb["value"] == d["value"] and cb["sample"]
    e2e = d["e2e"]
    assert e2e["value"] == d["value"] and e2e["unit"] == d["unit"]
    assert e2e["h2d_bytes_per_step"] == 0 and e2e["d2h_bytes_per_step"] == 0


def test_reference_arm_under_a_multi_rank_launch_only_rank_zero_prints():
    env = dict(os.environ, RANK="1", LOCAL_RANK="1", WORLD_SIZE="2", MASTER_ADDR="127.0.0.1", MASTER_PORT="29577")
    cmd = [sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "2", "--steps", "1",
           "--cpu-seconds", "1"]
    out = subprocess.run(cmd, cwd=ROOT, env=env, capture_output=True, text=True, timeout=300,
                         stdin=subprocess.DEVNULL)
    assert out.returncode == 0, out.stderr[-2000:]
    assert not [ln for ln in out.stdout.splitlines() if ln.startswith("{")]


def test_decode_roofline_names_the_kernel_that_the_step_launches():
    import bench
    from ffai_b200 import synth
    spec = synth.cfg2_gptoss()
    peaks = {"hbm_gbs": 6500.0, "source": "given"}
    one = bench.decode_roofline(spec, 1, 4.0, 0.03, None, peaks, {"dram": 1})
    assert one["kernel"] == "one_launch" and one["kernel_ms"] == 0.03 and "down" not in one and one["traffic"] is None
    assert one["algorithmic_bytes_per_launch"] == spec.decode_bytes(1, 4.0)
    chain = bench.decode_roofline(spec, 64, 32.0, 0.15, {"gate_up": 0.08, "down": 0.04}, peaks, {"dram": 1})
    assert chain["kernel"] == "gate_up" and chain["kernel_ms"] == 0.08 and chain["down"]["kernel_ms"] == 0.04 and chain["traffic"] == {"dram": 1}
