"""The build where the batch packer (gtd_pack.c) cannot be compiled, and its
library's name."""
import os
import subprocess
import sysconfig

import numpy as np
import pytest

from gisbdw_gb300 import _lib
from gisbdw_gb300 import build as B
from gisbdw_gb300 import graphs as G


@pytest.fixture(params=["no compiler", "no headers"])
def no_pack(request, monkeypatch, tmp_path):
    """An empty output folder; nvcc writes empty files, gcc is missing or fails."""
    for name, path in (("OUT_DIR", tmp_path), ("LIB", tmp_path / "libgtd.so"),
                       ("PACK_LIB", tmp_path / os.path.basename(B.PACK_LIB))):
        monkeypatch.setattr(B, name, str(path))

    def run(cmd, **kw):
        if os.path.basename(cmd[0]) == "gcc":
            if request.param == "no compiler":
                raise FileNotFoundError("gcc")
            return subprocess.CompletedProcess(cmd, 1, "", "Python.h: No such file or directory")
        open(cmd[cmd.index("-o") + 1], "w").close()
        return subprocess.CompletedProcess(cmd, 0, "", "")
    monkeypatch.setattr(B.subprocess, "run", run)


def test_build_goes_on_without_the_packer(no_pack):
    assert B.build(force=True) == B.LIB and os.path.exists(B.LIB)
    assert not os.path.exists(B.PACK_LIB) and B.up_to_date()


def test_batches_are_packed_without_the_packer(no_pack, monkeypatch):
    monkeypatch.setattr(_lib, "_PACK", None)
    monkeypatch.setattr(_lib, "load", lambda *a, **k: None)
    gs = [G.Graph(1, []), G.complete(64), G.grid(4, 5), G.cycle(64)]
    assert np.array_equal(_lib.adjacency_pool(gs, 1), np.concatenate([g.adj64() for g in gs]))
    assert np.array_equal(_lib.adjacency_pool(gs, 2), np.concatenate([g.adj128() for g in gs]))


def test_a_packer_of_an_older_source_is_not_kept(no_pack):
    open(B.PACK_LIB, "w").close()
    os.utime(B.PACK_LIB, (1, 1))
    assert B.pack_library() is None and not os.path.exists(B.PACK_LIB)


def test_the_packer_is_named_after_its_interpreter():
    assert B.PACK_LIB.endswith(sysconfig.get_config_var("EXT_SUFFIX"))
