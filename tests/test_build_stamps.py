"""What is rebuilt when: the extension module follows the interpreter and torch, the C library does not
need torch.  The compilers are replaced by recorders, nothing is compiled here."""
import subprocess
import sys
import types

import pytest

from ugache_b200 import build as b

torch = pytest.importorskip("torch")


@pytest.fixture
def recorder(tmp_path, monkeypatch):
    made = []

    def run(cmd, **kw):
        out = cmd[cmd.index("-o") + 1]
        made.append(out.rsplit("/", 1)[-1])
        open(out, "w").write("x")
        return types.SimpleNamespace(returncode=0, stderr="", stdout="")

    (tmp_path / "build").mkdir()
    monkeypatch.setattr(b, "HERE", str(tmp_path))
    monkeypatch.setattr(b, "LIB", str(tmp_path / "lib.so"))
    monkeypatch.setattr(b, "FAST", str(tmp_path / "_fast.so"))
    monkeypatch.setattr(b, "STAMP", str(tmp_path / "build" / "stamp.txt"))
    monkeypatch.setattr(b, "FAST_STAMP", str(tmp_path / "build" / "fast_stamp.txt"))
    monkeypatch.setattr(b.subprocess, "run", run)

    def build():
        made.clear()
        b.build()
        return sorted(x for x in made if x.endswith(".so"))

    return build


def test_another_torch_rebuilds_the_extension_only(recorder, monkeypatch):
    assert recorder() == ["_fast.so", "lib.so"]
    assert recorder() == []
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    assert recorder() == ["_fast.so"]
    assert recorder() == []


def test_without_torch_the_library_is_built_once(recorder, monkeypatch, capsys):
    monkeypatch.setitem(sys.modules, "torch", None)      # import torch raises ImportError
    assert recorder() == ["lib.so"]
    assert "torch" in capsys.readouterr().err
    assert recorder() == []


def test_a_failing_extension_keeps_the_library(recorder, monkeypatch):
    ok = b.subprocess.run
    monkeypatch.setattr(b.subprocess, "run", lambda cmd, **kw: types.SimpleNamespace(returncode=1, stderr="no", stdout="")
                        if cmd[0] == "g++" else ok(cmd, **kw))
    with pytest.raises(RuntimeError, match="g\\+\\+ failed"):
        recorder()
    monkeypatch.setattr(b.subprocess, "run", ok)
    assert recorder() == ["_fast.so"]


def test_a_module_of_another_torch_is_refused(built_lib):
    """In a process of its own: one that loads the module must not meet another torch afterwards."""
    code = ("import torch; torch.__version__ = '9.9.9'\n"
            "from ugache_b200 import _lib\n"
            "try:\n    _lib.fast()\nexcept ImportError as e:\n    print('refused', e)\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=b.os.path.dirname(b.HERE))
    assert "refused" in r.stdout and "9.9.9" in r.stdout, r.stdout + r.stderr
