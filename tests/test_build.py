"""The build from a checkout that has nothing built, in a copy of the package; nvcc is a stand-in that hands out the library built here."""
import os
import shutil
import subprocess
import sys
import sysconfig

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BUILT = os.path.join(ROOT, "dvm_b200", "lib", "libdvm_b200.so")
USE = """
import dvm_b200 as dvm
from dvm_b200 import _capi
r = dvm.IntArrayRef([1])
r.update([2, 3])
assert r.shape() == (2, 3)
k = dvm.PyKernel("vector", "das")
x = k.load([4, 64], dvm.float32)
k.store(k.add(x, x))
k.codegen()
assert "Add" in k.das()
"""
BUILD = "import __graft_entry__ as g\ng.build()\n"


@pytest.fixture
def tree(tmp_path):
    """(run, library folder): a copy of the sources with nothing built, and what runs a program in it."""
    skip = shutil.ignore_patterns("lib", "__pycache__")
    shutil.copytree(os.path.join(ROOT, "dvm_b200"), tmp_path / "dvm_b200", ignore=skip)
    shutil.copytree(os.path.join(ROOT, "include"), tmp_path / "include")
    shutil.copy(os.path.join(ROOT, "__graft_entry__.py"), tmp_path)
    nvcc = tmp_path / "cuda" / "bin" / "nvcc"
    nvcc.parent.mkdir(parents=True)
    nvcc.write_text("#!%s\nimport shutil, sys\nto = sys.argv[sys.argv.index('-o') + 1]\n"
                    "shutil.copy(%r, to) if '-shared' in sys.argv else open(to, 'w').close()\n" % (sys.executable, BUILT))
    nvcc.chmod(0o755)

    def run(program, **extra):
        env = {k: v for k, v in os.environ.items() if k != "PYTHONPATH"}
        env.update({"CUDA_HOME": str(tmp_path / "cuda")}, **extra)
        r = subprocess.run([sys.executable, "-c", program], cwd=tmp_path, env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout + r.stderr

    return run, tmp_path / "dvm_b200" / "lib"


def test_a_checkout_is_built_and_used_in_one_process(tree):
    run, _ = tree
    run(BUILD + USE + "assert hasattr(_capi.calls, 'setup')   # (the extension module, not what stands for it)")
    run(USE)


def test_the_build_imports_nothing_that_it_makes(tree):
    run, _ = tree
    run("import sys, dvm_b200.build as b\nassert 'dvm_b200._capi' not in sys.modules\nb.build()\n" + USE)


@pytest.mark.parametrize("content", [b"", b"\x7fELF", b"no library"])
def test_a_damaged_extension_module_is_built_anew(tree, content):
    run, lib = tree
    run(BUILD)
    (module,) = lib.glob("_calls*")
    size = module.stat().st_size
    module.write_bytes(content)
    run(BUILD + USE)
    assert module.stat().st_size == size and list(lib.glob("_calls*")) == [module]
    assert run("import dvm_b200.build as b\nb._nvcc = None\nb.subprocess = None\nb.build()") == ""   # (nothing is left to do)


def test_the_extension_module_follows_the_c_abi(tree):
    """A change of the C ABI's header builds the module anew, and one that its calls do not fit is an error of the compiler."""
    run, lib = tree
    run(BUILD)
    (module,) = lib.glob("_calls*")
    header = lib.parent.parent / "include" / "dvm_c.h"
    at = module.stat().st_mtime
    os.utime(header, (at + 5, at + 5))
    os.utime(module, (at, at))
    run(BUILD + USE)
    assert module.stat().st_mtime != at
    text, launch = header.read_text(), "int dvm_launch(dvm_kernel *k, void *stream);"
    assert launch in text
    header.write_text(text.replace(launch, "int dvm_launch(dvm_kernel *k, void *stream, int priority);"))
    at = module.stat().st_mtime
    os.utime(header, (at + 5, at + 5))
    assert "too few arguments" in run(BUILD + USE) and not module.exists()


def test_without_the_headers_of_python(tree):
    """The library is made, an extension module of before does not stay, and the general methods do the module's work."""
    run, lib = tree
    gxx = lib.parent.parent / "bin" / "g++"
    gxx.parent.mkdir()
    gxx.write_text("#!/bin/sh\necho 'fatal error: Python.h: No such file or directory' >&2\nexit 1\n")
    gxx.chmod(0o755)
    lib.mkdir()
    (lib / ("_calls" + sysconfig.get_config_var("EXT_SUFFIX"))).write_bytes(b"of other sources")
    path = str(gxx.parent) + os.pathsep + os.environ["PATH"]
    assert "Python.h" in run(BUILD + USE, PATH=path)
    assert (lib / "libdvm_b200.so").exists() and not list(lib.glob("_calls*"))
    shutil.copy(os.path.join(ROOT, "tests", "test_calls.py"), lib.parent.parent)
    run("import pytest, sys\nfrom dvm_b200 import _capi\nassert _capi.calls is _capi._GeneralCalls\n"
        "sys.exit(pytest.main(['-q', '-p', 'no:cacheprovider', 'test_calls.py']))")


def test_graphs_of_others_load_nothing_of_this_library():
    """workloads builds its graphs on whatever kernel object it is given (the benchmark's reference arm gives it the reference's)."""
    code = "import dvm_b200.workloads\nassert not [l for l in open('/proc/self/maps') if 'dvm_b200/lib' in l]"
    assert subprocess.run([sys.executable, "-c", code], cwd=ROOT).returncode == 0


def test_names_of_the_package():
    import dvm_b200
    for name in dvm_b200.__all__:
        assert getattr(dvm_b200, name) is not None and name in dir(dvm_b200)
    assert dvm_b200.float16 is dvm_b200.frontend.DataType.float16 and dvm_b200.kernel is dvm_b200.jit.kernel
    with pytest.raises(AttributeError):
        dvm_b200.no_such_name
