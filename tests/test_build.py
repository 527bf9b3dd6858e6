"""What the Python front end's extension is built from, and how a build that does not fit shows."""
import subprocess
import sys
from pathlib import Path

from autograph_b200 import build

ROOT = Path(__file__).resolve().parent.parent


def _run(code):
    res = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=ROOT)
    assert res.returncode == 0, res.stderr[-3000:]


def test_another_torch_version_rebuilds_the_extension(tmp_path):
    (tmp_path / "version.py").write_text("__version__ = '2.11.0'\n")
    cmd, key = build._front_recipe(tmp_path)
    assert build._front_recipe(tmp_path) == (cmd, key)
    (tmp_path / "version.py").write_text("__version__ = '2.12.0'\n")
    assert build._front_recipe(tmp_path)[0] == cmd and build._front_recipe(tmp_path)[1] != key


def test_an_extension_that_does_not_load_says_why():
    """The package still imports (the build imports it); the import's own error is in the one that a device raises."""
    _run("""
import sys
sys.modules["autograph_b200._front"] = None   # importing it raises ImportError with this module's name
import autograph_b200 as ag
try:
    ag.Device
    ag._bind_front()
except ImportError as e:
    assert "halted" in str(e) and "autograph_b200.build" in str(e), e
    assert isinstance(e.__cause__, ImportError)
else:
    raise AssertionError("no error")
""")
