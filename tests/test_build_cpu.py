"""build.py rebuilds the PyTorch extension for another PyTorch, Python or command, and not otherwise."""
import importlib.util
import os
import sys

import torch

from tests.conftest import ROOT


def test_the_extension_is_rebuilt_for_another_torch_or_python(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location('fwp_build', os.path.join(ROOT, 'recurrent_fwp_b200', 'build.py'))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    src, so, stamp = (str(tmp_path / n) for n in ('binding.cpp', 'binding.so', 'stamp'))
    for name, value in (('BINDING_SRC', src), ('BINDING', so), ('BINDING_STAMP', stamp), ('PKG', str(tmp_path / 'pkg'))):
        monkeypatch.setattr(build, name, value)
    open(src, 'w').close()
    compiled = []

    class Done:
        returncode, stdout, stderr = 0, '', ''

    def compiler(cmd, **_):
        compiled.append(cmd)
        open(so, 'w').close()
        return Done

    monkeypatch.setattr(build.subprocess, 'run', compiler)
    assert build._binding_stale()               # nothing built yet
    build._compile_binding()
    assert len(compiled) == 1 and not build._binding_stale()
    with monkeypatch.context() as m:
        m.setattr(torch, '__version__', '0.0.0')
        assert build._binding_stale()
    with monkeypatch.context() as m:
        m.setattr(sys, 'version', 'another')
        assert build._binding_stale()
    with monkeypatch.context() as m:
        m.setenv('CXX', 'another-compiler')
        assert build._binding_stale()
    assert not build._binding_stale()
    os.remove(stamp)
    assert build._binding_stale()
