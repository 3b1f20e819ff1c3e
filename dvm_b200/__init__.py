"""dvm_b200: B200-native device virtual machine for fused tensor operators.

Drop-in for the fused-operator path of mindspore-ai/dvm: the package exports the names of the reference's
``dvm`` Python package (python/dvm/__init__.py:17-42) - DataType, Device, Kernel, PyKernel, NDObject,
IntArrayRef, ScalarRef, the dtype aliases and the ``kernel`` decorator - implemented over the C ABI of
``libdvm_b200.so`` (include/dvm_c.h).

The front-end is imported with the first name that is taken from it, not with the package: ``dvm_b200.build`` lies in this
package too, and must not load what it is about to make.
"""
import importlib

_TYPES = {"bool_": "bool", "float16": "float16", "bfloat16": "bfloat16", "float32": "float32", "int32": "int32", "int64": "int64"}
_HOME = {"kernel": "jit", "JitKernel": "jit"}   # of names that are not the front-end's

__all__ = [
    "DataType", "Device", "Kernel", "PyKernel", "NDObject", "IntArrayRef", "ScalarRef", "DvmError",
    "kernel", "JitKernel", "bool_", "float16", "bfloat16", "float32", "int32", "int64",
]


def __getattr__(name):
    if name in ("_capi", "frontend", "jit"):
        return importlib.import_module("." + name, __name__)
    if name not in __all__:
        raise AttributeError("module %r has no attribute %r" % (__name__, name))
    module = importlib.import_module("." + _HOME.get(name, "frontend"), __name__)
    value = getattr(module.DataType, _TYPES[name]) if name in _TYPES else getattr(module, name)
    globals()[name] = value
    return value


def __dir__():
    return sorted(set(globals()) | set(__all__))
