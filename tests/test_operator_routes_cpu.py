"""The operators of ops/nodes.py without their native nodes: nothing built and no compiler, or a torch without the interfaces they use."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import test_operators_cpu as native_tests

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("have_private", [True, False])
@pytest.mark.parametrize("name", ["test_transforms", "test_vmap_of_leaves_that_autograd_follows", "test_autograd_and_what_it_saves", "test_refused",
                                  "test_outputs_that_the_loss_does_not_use", "test_text_argument_and_saved_outputs"])
def test_python_functions_do_the_same(name, have_private, monkeypatch):
    from opake_b200.ops import nodes

    monkeypatch.setattr(nodes, "_NATIVE", False)
    monkeypatch.setattr(nodes, "_HAVE_PRIVATE", have_private)
    test = getattr(native_tests, name)
    for mark in getattr(test, "pytestmark", []):
        for transform in mark.args[1]:
            test(transform)
    if not getattr(test, "pytestmark", []):
        test()


def test_without_library_and_compiler(tmp_path):
    """Importing works, what nothing differentiates runs, and what autograd follows falls back with one warning."""
    code = """
import warnings
from pathlib import Path
from opake_b200 import _build
_build.OUT = Path(%r)
warnings.simplefilter("error")
import torch
import opake_b200.patches, opake_b200.patches.kernels, opake_b200.ops.lce, opake_b200.alignment.logprob, opake_b200.alignment.sft.loss
from opake_b200.patches.kernels import lora_linear, opake_rms_norm, opake_swiglu
x, w, a, b = (torch.randn(s, dtype=torch.float64) for s in ((4, 6), (5, 6), (2, 6), (5, 2)))
opake_rms_norm(x, x[0]), opake_swiglu(x, x)
assert torch.allclose(lora_linear(x, w, a, b, 0.5), x @ w.t() + 0.5 * (x @ a.t()) @ b.t())
loss = lambda a, x: lora_linear(x, w, a, b, 0.5).pow(2).sum()
plain = lambda a, x: (x @ w.t() + 0.5 * (x @ a.t()) @ b.t()).pow(2).sum()
per = lambda f: torch.func.vmap(torch.func.grad(f), (None, 0))(a, x[:, None])
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    got, again = per(loss), per(loss)
assert torch.allclose(got, per(plain)) and torch.equal(got, again)
assert sum("native autograd nodes" in str(s.message) for s in seen) == 1, [str(s.message) for s in seen]
print("fell back")
""" % str(tmp_path)
    run = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env={**os.environ, "CXX": "/nonexistent/compiler"}, capture_output=True, text=True)
    assert run.returncode == 0 and "fell back" in run.stdout, run.stderr[-2000:]


def test_library_of_another_torch_or_source_is_not_taken(tmp_path, monkeypatch):
    import torch

    from opake_b200 import _build

    name = _build.nodes_lib().name
    monkeypatch.setattr(torch, "__version__", "9.9.9+other")
    other_torch = _build.nodes_lib().name
    monkeypatch.undo()
    (tmp_path / "host").mkdir()
    (tmp_path / "host" / "nodes.cpp").write_bytes((_build.CSRC / "host" / "nodes.cpp").read_bytes() + b"\n")
    monkeypatch.setattr(_build, "CSRC", tmp_path)
    assert len({name, other_torch, _build.nodes_lib().name}) == 3


@pytest.mark.parametrize("status", [0, 1])
def test_library_appears_whole(tmp_path, monkeypatch, status):
    """While the compiler writes, nothing stands where the library will be; a failed build leaves nothing behind."""
    from opake_b200 import _build

    monkeypatch.setattr(_build, "OUT", tmp_path / "out")
    seen = tmp_path / "seen"
    compiler = tmp_path / "cxx"
    compiler.write_text(f'''#!{sys.executable}
import os, sys
out = sys.argv[sys.argv.index("-o") + 1]
open(out, "w").write("half")
open({str(seen)!r}, "w").write(str(os.path.exists({str(_build.nodes_lib())!r})))
open(out, "a").write(" and half")
sys.exit({status})
''')
    compiler.chmod(0o755)
    monkeypatch.setenv("CXX", str(compiler))
    if status:
        with pytest.raises(RuntimeError, match="build of the autograd nodes failed"):
            _build.build_nodes()
        assert not list((tmp_path / "out").iterdir())
    else:
        path = _build.build_nodes()
        assert path.read_text() == "half and half" and list((tmp_path / "out").iterdir()) == [path]
    assert seen.read_text() == "False"
