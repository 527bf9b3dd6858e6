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


def test_the_library_needs_no_torch():
    """Hosts in C and Rust build the library, and Python hosts may call it through ctypes, without torch."""
    _run("""
import sys
sys.modules["torch"] = None
import autograph_b200 as ag
assert ag.lib().ag_kernel_launch_count and ag.kernel_launch_count() == 0
try:
    ag.Device(0)
except ImportError as e:
    assert "torch" in str(e)
else:
    raise AssertionError("no error")
""")
    _run("import sys, autograph_b200; assert 'torch' not in sys.modules")
    _run("""
from autograph_b200 import *
from autograph_b200 import _front, _PyDevice, _PyModel
assert Device.__mro__[1:3] == (_front.DeviceBase, _PyDevice) and Model.__mro__[1:3] == (_front.ModelBase, _PyModel)
assert Device.__doc__ == _PyDevice.__doc__ and Device.__module__ == "autograph_b200"
""")


def test_the_library_is_built_first_and_without_torch(monkeypatch, tmp_path, capsys):
    import importlib.util
    monkeypatch.setattr(importlib.util, "find_spec", lambda name: None)
    assert build.build_front() is None
    order = []
    monkeypatch.setattr(build, "BUILD", tmp_path)
    monkeypatch.setattr(build, "LIB", tmp_path / "library.so")
    monkeypatch.setattr(build, "_compile", lambda src, *a: order.append("library") or Path(__file__))
    monkeypatch.setattr(build, "build_front", lambda force=False: order.append("front"))
    monkeypatch.setattr(build.subprocess, "run", lambda *a, **k: type("Done", (), {"returncode": 0}))
    assert build.build() == build.LIB
    assert order[-1] == "front" and order.count("front") == 1 and "without the Python front end" in capsys.readouterr().err
