"""Launches over rows without a column: nothing to do, and no division by the width on the way there (it would end the process)."""
import subprocess
import sys

CALLS = ["norm(z, z, z, z, z, z, z, 0, 4, 0, 1e-5, 0, z)", "act_mul(z, z, z, z, 0, 4, 0, 0, 0, 1, z, z)", "quant_fp8(z, z, z, 4, 4, 0, 0, z)",
         "quant_nvfp4(z, 0, z, 0, z, 0, z, 4, 0, z)",
         "rope_kv_append(z, z, 0, z, z, z, 0, 16, 4, 8, 2, 0, 0, 1, 0, 0, 0, 1.0, 1.0, 1, z)",        # no columns
         "rope_kv_append(z, z, 0, z, z, z, 0, 16, 4, 0, 0, 128, 128, 1, 0, 0, 0, 1.0, 1.0, 1, z)"]    # no heads


def test_rows_without_columns():
    code = "from ksanallm_b200.ops import native; z = None; lib = native._load()\n"
    code += "".join(f"print({c[:4]!r}, lib.ksana_{c}, flush=True)\n" for c in CALLS)
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and done.stdout.splitlines() == [f"{c[:4]} 0" for c in CALLS], (done.returncode, done.stdout)
