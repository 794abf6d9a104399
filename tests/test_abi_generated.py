"""include/vta_gb300.h and the other generated files are what gen_abi.py writes."""
import os
import shutil
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_generated_files_match_their_generator(tmp_path):
    for d in ("include", "vectorta_gb300/csrc", "vectorta_gb300/rust"):
        shutil.copytree(os.path.join(ROOT, d), tmp_path / d)
    subprocess.run([sys.executable, "vectorta_gb300/csrc/gen_abi.py"], cwd=tmp_path, check=True, capture_output=True)
    for f in ("include/vta_gb300.h", "vectorta_gb300/csrc/vta_abi_gen.inc", "vectorta_gb300/rust/vta_sys/src/lib.rs"):
        assert (tmp_path / f).read_text() == open(os.path.join(ROOT, f)).read(), f
