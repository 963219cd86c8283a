"""A changed source of any kind makes the built library stale."""
import os

import pytest

from pyheadtail_gb300 import _build


@pytest.mark.parametrize('suffix', ['.cu', '.cuh', '.h', '.inc'])
def test_newer_source_is_stale(suffix, tmp_path, monkeypatch):
    csrc = tmp_path / 'csrc'
    csrc.mkdir()
    lib = tmp_path / 'libphk.so'
    src = csrc / ('part' + suffix)
    src.write_text('')
    lib.write_text('')
    for k, v in (('CSRC', csrc), ('INCLUDE', csrc), ('LIB', lib)):
        monkeypatch.setattr(_build, k, str(v))
    t = os.path.getmtime(_build.__file__)
    os.utime(lib, (t + 10, t + 10))
    os.utime(src, (t + 5, t + 5))
    assert not _build._stale()
    os.utime(src, (t + 20, t + 20))
    assert _build._stale()
