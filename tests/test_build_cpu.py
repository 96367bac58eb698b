"""The rule that decides when the extension module is compiled again, on stand-ins for the compiler."""
import subprocess

import torch

from brainpylib_b200 import build


def test_native_module_is_rebuilt_for_another_torch(tmp_path, monkeypatch):
  commands = []

  def compiler(cmd, **kwargs):
    commands.append(cmd)
    open(cmd[cmd.index('-o') + 1], 'w').close()
    return subprocess.CompletedProcess(cmd, 0, stdout='')

  monkeypatch.setattr(build, 'NATIVE', str(tmp_path / '_native.so'))
  monkeypatch.setattr(build, 'BUILD_DIR', str(tmp_path))
  monkeypatch.setattr(build, 'NATIVE_STAMP', str(tmp_path / 'native_torch.txt'), raising=False)
  monkeypatch.setattr(build.subprocess, 'run', compiler)
  build._build_native(False, False)
  build._build_native(False, False)
  assert len(commands) == 1
  monkeypatch.setattr(torch, '__version__', '0.0.1')
  build._build_native(False, False)
  assert len(commands) == 2
  monkeypatch.setattr(build.os, 'getpid', lambda: 12345)
  build._build_native(True, False)
  targets = [c[c.index('-o') + 1] for c in commands]
  assert targets[2] != targets[1] and build.NATIVE not in targets      # a name of its own per process
