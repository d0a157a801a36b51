"""The built package works from where it lies, not from where it was built."""
import os
import shutil
import subprocess
import sys

import vulkanforge_b200 as vf


def test_bindings_load_the_library_beside_them(tmp_path):
    vf.load()
    package = os.path.dirname(os.path.abspath(vf.__file__))
    moved = tmp_path / "elsewhere" / "vulkanforge_b200"
    shutil.copytree(package, moved, ignore=shutil.ignore_patterns("csrc", "build", "__pycache__"))
    code = ("import vulkanforge_b200._lib as l; l.native(); "
            "print('\\n'.join(sorted({x.split()[-1] for x in open('/proc/self/maps') if 'libvfkv.so' in x})))")
    env = {k: v for k, v in os.environ.items() if k != "PYTHONPATH"}
    out = subprocess.run([sys.executable, "-c", code], cwd=moved.parent, env=env, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert out.stdout.split() == [str(moved / "libvfkv.so")]
