"""How the library is split into modules (no GPU): the CUDA runtime loads a module whole at its first launch, so the variants of a
kernel that one process hardly ever needs together are separate objects."""
import os
import shutil
import subprocess

import pytest

from pink_b200 import build


def test_rotation_variants_are_separate_modules():
    names = [name for name, _, _ in build.VARIANTS]
    assert len(set(names)) == len(names) == 10 and all(src == "rotate.cu" for _, src, _ in build.VARIANTS)
    objdir = os.path.join(build.HERE, "build")
    if not os.path.isdir(objdir) or not shutil.which("nm"):
        pytest.skip("no object files")
    for name in names + ["rotate"]:
        obj = os.path.join(objdir, name + ".o")
        symbols = subprocess.run(["nm", "-C", obj], capture_output=True, text=True, check=True).stdout.splitlines()
        kernels = {s[19:] for s in symbols if "::rotate_kernel<" in s and "__device_stub" not in s}
        assert len(kernels) == 0 if name == "rotate" else 1 <= len(kernels) <= 5, (name, len(kernels))
