"""The in-tree build: without PyTorch, after a PyTorch upgrade, and called by several processes or threads at once."""
import importlib.util
import threading
import time
from pathlib import Path

import pytest

from aluminum_b200 import _build


@pytest.fixture
def fake(monkeypatch, tmp_path):
    """The build with every command replaced by one that writes its output file; yields the commands."""
    for name, path in (("OBJ", "obj"), ("LIB", "lib/libal_b200.so"), ("TORCH_LIB", "lib/libal_torch.so"), ("BIN", "bin")):
        monkeypatch.setattr(_build, name, tmp_path / path)
    commands, running, lock = [], [0, 0], threading.Lock()

    def run(cmd):
        link = "-shared" in cmd
        with lock:
            commands.append(cmd)
            running[0] += link
            running[1] = max(running)
        time.sleep(0.02 if link else 0)
        Path(cmd[cmd.index("-o") + 1]).write_text("x")
        with lock:
            running[0] -= link
    monkeypatch.setattr(_build, "_run", run)
    monkeypatch.setattr(_build.shutil, "which", lambda name: name)
    commands_of = lambda part: [c for c in commands if any(part in str(a) for a in c)]
    yield commands, commands_of, running


def test_without_pytorch(fake, monkeypatch):
    commands, commands_of, _ = fake
    find = importlib.util.find_spec
    monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
    assert _build._torch_dir() is None
    assert _build.build(tools=False).exists() and not _build.TORCH_LIB.exists()
    assert commands_of("libal_b200") and not commands_of("src/torch")


def test_operators_follow_the_installed_pytorch(fake, monkeypatch):
    commands, commands_of, _ = fake
    _build.build(tools=False)
    assert _build.TORCH_LIB.exists() and commands_of("src/torch")
    commands.clear()
    _build.build(tools=False)
    assert not commands
    monkeypatch.setattr(_build, "_torch_stamp", lambda: "another version")
    _build.build(tools=False)
    assert len(commands_of("src/torch")) == 1 and len(commands) == 2   # the operators are compiled and linked again, nothing else


def test_one_build_at_a_time(fake):
    commands, commands_of, running = fake
    threads = [threading.Thread(target=_build.build, kwargs=dict(tools=False)) for _ in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert running[1] == 1 and len([c for c in commands if "-shared" in c]) == 2
    assert not list(_build.LIB.parent.glob(".*"))   # complete files only
