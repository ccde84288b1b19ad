"""bench.py's reference arm on CPU: one JSON line with the contract's keys from
rank 0, nothing from the other ranks. (The GPU arm needs a device.)"""

from __future__ import annotations

import json
import os
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def run_reference_arm(env_extra: dict) -> subprocess.CompletedProcess:
    env = dict(os.environ, **env_extra)
    return subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "2", "--warmup", "3"],
                          cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)


def test_reference_arm_prints_one_contract_line():
    done = run_reference_arm({"RANK": "0"})
    assert done.returncode == 0, done.stderr[-2000:]
    lines = [line for line in done.stdout.splitlines() if line.startswith("{")]
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert line["impl"] == "reference"
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
                "scaling", "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e"):
        assert key in line, key
    assert line["steps"] == 2 and line["warmup"] == 3 and line["n_gpus"] == 1
    assert line["value"] > 0 and line["higher_is_better"] is True
    assert line["config"]["workload"] == "2d_type1_modes1024x1024_M1e7_uniform_eps1e-5"
    cpu = line["cpu_baseline"]
    assert cpu["kind"] in ("port", "reference") and cpu["cores"] >= 1 and cpu["value"] == line["value"]
    assert cpu["unit"] == line["unit"] and cpu["sample"]
    e2e = line["e2e"]
    assert e2e["value"] == line["value"] and e2e["unit"] == line["unit"]
    assert e2e["h2d_bytes_per_step"] == 0 and e2e["d2h_bytes_per_step"] == 0


def test_reference_arm_other_ranks_exit_quietly():
    done = run_reference_arm({"RANK": "1"})
    assert done.returncode == 0, done.stderr[-2000:]
    assert not [line for line in done.stdout.splitlines() if line.startswith("{")]


def test_the_json_line_is_short_and_whole():
    """A reader that keeps the last 3,000 characters of the output gets the whole line."""
    sys.path.insert(0, str(ROOT))
    import bench

    number, text = 12345678901.234567, "x" * 300
    line = {k: number for k in bench.LINE_KEYS}
    line.update(metric=bench.METRIC, data=text[:60], config={k: text[:60] for k in "abcdefgh"},
                e2e={"value": number, "unit": "points/s", "ms_per_step": number, "h2d_bytes_per_step": 160000000,
                     "d2h_bytes_per_step": 8388608, "path": text},
                clocks={"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": [], "samples": 2},
                roofline={**{k: number for k in "abcdefg"}, "traffic_source": text, "peak_source": text[:60]},
                cpu_baseline={"value": number, "sample": text, "one_shot_value": number})
    line.update(batched={"entries": [text] * 100}, type2={"value": number, "rel_l2": 1e-5, "stages": text},
                one_shot={"value": number}, summary={"all": text})
    details, short = bench.split_line(line)
    assert len(json.dumps(short, separators=(",", ":"))) < 2_900
    assert set(bench.LINE_KEYS) <= set(short) and short["type2"]["value"] > 0
    assert set(details) | set(short) >= set(line) and "batched" in details
