"""When the extension module is built again: for another torch or Python, with that torch's ABI; and that one for another torch
is not used."""
import pytest
import torch

from adacode_b200 import _lib, build


@pytest.fixture
def compiled(monkeypatch):
    """Compiler commands that a build would run."""
    commands = []
    monkeypatch.setattr(build, '_run', lambda cmd: commands.append(cmd) or '')
    return commands


def test_an_up_to_date_module_is_kept(compiled):
    build.build_native()
    assert compiled == []


def test_another_torch_is_another_module(compiled, monkeypatch):
    monkeypatch.setattr(torch, '__version__', '9.9.9+test')
    build.build_native()
    assert len(compiled) == 1


def test_another_python_is_another_file(monkeypatch):
    import sysconfig
    assert build.native_path().endswith('_native' + sysconfig.get_config_var('EXT_SUFFIX'))


def test_the_abi_is_torchs(compiled):
    build.build_native(force=True)
    assert f'-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}' in compiled[0]


def test_a_module_for_another_torch_is_refused(monkeypatch):
    _lib.native()
    monkeypatch.setattr(_lib, '_native', None)
    monkeypatch.setattr(torch, '__version__', '9.9.9+test')
    with pytest.raises(_lib.AdacodeError, match='adacode_b200.build'):
        _lib.native()
