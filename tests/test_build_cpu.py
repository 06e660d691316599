"""The two shared libraries when one of them is missing, unusable, built for another torch or already in use: importing the
package works, a call says what to do, and a build repairs the state.  The compilers are stand-ins that hand out the real libraries."""

import os
import shutil
import stat
import subprocess
import sys
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NAMES = ("libkda_b200.so", "libkda_b200_torch.so")


@pytest.fixture
def tree(tmp_path):
    """A copy of the package with its libraries; its compilers copy what `finished` holds to their -o argument."""
    import __graft_entry__  # noqa: F401  (path setup)
    from kda_b200 import build

    build.build()
    for part in ("include", "attention-gym_b200"):
        shutil.copytree(os.path.join(ROOT, part), tmp_path / part)
    package = tmp_path / "attention-gym_b200" / "kda_b200"
    finished = tmp_path / "finished"
    finished.mkdir()
    for name in NAMES:
        shutil.copy(package / name, finished / name)
    compiler = tmp_path / "compiler"
    compiler.write_text(textwrap.dedent(f"""\
        #!/bin/sh
        while [ $# -gt 0 ]; do
          if [ "$1" = -o ]; then out=$2; fi
          shift
        done
        case "$out" in
          *.so) cp "{finished}/$(basename "$out")" "$out";;
          *) : > "$out";;
        esac
        """))
    compiler.chmod(compiler.stat().st_mode | stat.S_IXUSR)
    env = dict(os.environ, NVCC=str(compiler), CXX=str(compiler), PYTHONPATH=str(package.parent))

    def run(*args):
        return subprocess.run([sys.executable, *args], env=env, cwd=tmp_path, capture_output=True, text=True)

    return package, run


CALL = """
import torch, kda_b200
from kda_b200 import _cabi
assert not _cabi.mapped()
try:
    _cabi.load_torch_library()
    print("loaded", torch._C._dispatch_has_kernel_for_dispatch_key("kda_b200::kda_chunk_fwd", "CUDA"))
except RuntimeError as error:
    print("refused", error)
"""


@pytest.mark.parametrize("name", NAMES)
def test_missing_library(tree, name):
    package, run = tree
    os.remove(package / name)
    said = run("-c", CALL)
    assert said.returncode == 0 and "refused" in said.stdout and "is missing: build it" in said.stdout, said.stderr
    built = run("-m", "kda_b200.build")
    assert built.returncode == 0, built.stderr
    assert "loaded True" in run("-c", CALL).stdout


def test_unusable_operator_library(tree):
    package, run = tree
    (package / NAMES[1]).write_bytes(b"not a library")
    said = run("-c", CALL)
    assert said.returncode == 0 and "cannot be loaded" in said.stdout and "--force" in said.stdout, said.stderr
    built = run("-m", "kda_b200.build", "--force")
    assert built.returncode == 0, built.stderr
    assert "loaded True" in run("-c", CALL).stdout


def test_another_torch(tree):
    package, run = tree
    check = "from kda_b200 import build; print(build.needs_build())"
    assert run("-c", check).stdout.strip() == "False"
    (package / "_obj" / "torch_build").write_text("1.0 cxx11=0")
    assert run("-c", check).stdout.strip() == "True"
    assert run("-m", "kda_b200.build").returncode == 0
    assert run("-c", check).stdout.strip() == "False"


def test_a_failed_build_leaves_the_old_libraries(tree):
    package, run = tree
    before = [(package / n).read_bytes() for n in NAMES]
    os.remove(package.parent.parent / "finished" / NAMES[1])       # linking the second library fails
    assert run("-m", "kda_b200.build", "--force").returncode != 0
    assert [(package / n).read_bytes() for n in NAMES] == before
    assert "loaded True" in run("-c", CALL).stdout


def test_a_library_in_use(tree):
    _, run = tree
    said = run("-c", "import kda_b200\nfrom kda_b200 import _cabi, build\nbuild.build(force=True)\nprint('first')\n"
                     "_cabi.lib()\nbuild.build(force=True)")
    assert "first" in said.stdout and said.returncode != 0 and "restart it" in said.stderr


def test_operators_refuse_cpu_tensors_as_before():
    import torch

    import __graft_entry__  # noqa: F401  (path setup)
    import kda_b200  # noqa: F401

    x = torch.zeros(1, 64, 1, 128, dtype=torch.bfloat16)
    with pytest.raises(NotImplementedError, match="Could not run 'kda_b200::kda_chunk_fwd'"):
        torch.ops.kda_b200.kda_chunk_fwd(x, x, x, x.float(), x[..., 0].float(), None, True)


def test_a_refusal_whose_message_holds_a_number():
    """An exception of the operator library with a formatted number, in a process of its own: it must not crash.  (The CUDA
    implementation is called with CPU tensors; it refuses them before it touches one.)"""
    import __graft_entry__  # noqa: F401  (path setup)
    from kda_b200 import build

    build.build()
    said = subprocess.run([sys.executable, "-c", textwrap.dedent("""\
        import torch, kda_b200
        from kda_b200 import _cabi
        _cabi.load_torch_library()
        q = torch.zeros(1, 64, 2, 128, dtype=torch.bfloat16)
        gate, beta, tape = torch.zeros(1, 64, 2, 128), torch.zeros(1, 64, 2), torch.zeros(1, 64, 2, 64, dtype=torch.bfloat16)
        saved, offsets = torch.zeros(2 ** 20, dtype=torch.uint8), torch.zeros(1, dtype=torch.int32)      # no sequence at all
        cuda = torch._C.DispatchKeySet(torch._C.DispatchKey.CUDA)
        try:
            torch.ops.kda_b200.kda_chunk_bwd_saved.default.redispatch(
                cuda, q, q, q, gate, beta, tape, tape, saved, offsets, offsets, None, None, None, False)
        except ValueError as error:
            print("refused:", error)
        """)], env=dict(os.environ, PYTHONPATH=os.path.join(ROOT, "attention-gym_b200")), capture_output=True, text=True)
    assert "refused: num_sequences must be positive, got 0" in said.stdout, (said.returncode, said.stderr[-500:])
