"""build() makes the product from the product's own files: no tests directory, no other checkout state."""
import os
import shutil
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_build_needs_no_tests_directory(tmp_path):
    for d in ("include", "orkan_b200"):     # with the objects, whose times make the build incremental
        shutil.copytree(os.path.join(ROOT, d), tmp_path / d, copy_function=shutil.copy2)
    shutil.copy2(os.path.join(ROOT, "__graft_entry__.py"), tmp_path)
    lib = tmp_path / "orkan_b200" / "liborkan_b200.so"
    if lib.exists():
        lib.unlink()                        # at least the link step runs
    env = {k: v for k, v in os.environ.items() if k not in ("PYTHONPATH", "ORKAN_REFERENCE_SRC")}
    r = subprocess.run([sys.executable, "-c", "import __graft_entry__ as g; g.build()"], cwd=tmp_path, env=env,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert lib.exists()
    assert not (tmp_path / "tests").exists()
