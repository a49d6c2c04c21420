"""The kernel build helper, as far as it goes without a GPU or a compiler run."""
import os
import re
from concurrent.futures import ThreadPoolExecutor

import pytest

from infernum_b200.csrc import build


def test_build_dir_from_many_threads(tmp_path, monkeypatch):
    """Modules are compiled from several threads at once; each of them asks for
    the folder, and none may be sent elsewhere because another one's probe file
    came and went."""
    target = tmp_path / "kernels"
    monkeypatch.setenv("INFERNUM_BUILD_DIR", str(target))
    with ThreadPoolExecutor(max_workers=16) as pool:
        dirs = list(pool.map(lambda _: build.build_dir(), range(300)))
    assert set(dirs) == {str(target)}
    assert [p.name for p in target.iterdir()] == []  # no probe file is left behind


def test_module_hash_follows_sources_and_flags():
    a = build._hash_module(["elementwise.cu"], [], "nvcc")
    assert a == build._hash_module(["elementwise.cu"], [], "nvcc")
    assert a != build._hash_module(["elementwise.cu"], ["-DIB_HD=64"], "nvcc")
    assert a != build._hash_module(["sampling.cu"], [], "nvcc")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(build.CSRC_DIR) if f.endswith(".cu")))
def test_no_thread_leaves_a_kernel_begun_early_without_waiting(name):
    """Between a kernel's ``pdl_trigger()`` and its first ``pdl_wait()`` nothing returns: a grid whose CTAs all left there
    would be complete before the grids before it are, and the kernel behind it would begin on what they still write."""
    with open(os.path.join(build.CSRC_DIR, name), encoding="utf-8") as fh:
        source = re.sub(r"//[^\n]*", "", fh.read())
    for m in re.finditer(r"pdl_trigger\(\);", source):
        before = source[m.end():].split("pdl_wait();")[0]
        assert not re.search(r"\breturn;", before), f"{name}: line {source.count(chr(10), 0, m.start()) + 1}"
