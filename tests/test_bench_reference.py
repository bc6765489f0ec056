"""bench.py's reference arm where the reference's library can be neither found
nor built: one line that says so, and exit code 0."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_unavailable_reference_is_one_line(tmp_path):
    # A copy of what the arm imports, without the reference's library; the
    # oracle looks for the sources in a folder that is not there.
    for f in ("bench.py", "oracle", "harmony_b200"):
        os.symlink(os.path.join(ROOT, f), tmp_path / f)
    os.unlink(tmp_path / "oracle")
    os.mkdir(tmp_path / "oracle")
    for f in os.listdir(os.path.join(ROOT, "oracle")):
        if f not in ("_ref", "__pycache__"):
            os.symlink(os.path.join(ROOT, "oracle", f), tmp_path / "oracle" / f)
    run = ("import sys, runpy, oracle; oracle.REFERENCE_SRC = sys.argv[1]; "
           "sys.argv = ['bench.py', '--impl', 'reference', '--gpus', '1', '--steps', '2', '--warmup', '3']; "
           "runpy.run_path('bench.py', run_name='__main__')")
    out = subprocess.run([sys.executable, "-c", run, str(tmp_path / "none")], cwd=tmp_path, capture_output=True, text=True,
                         timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    lines = [json.loads(line) for line in out.stdout.splitlines() if line.startswith("{")]
    assert len(lines) == 1 and lines[0]["impl"] == "reference" and "\n" not in lines[0]["unavailable"]
    assert "value" not in lines[0]
