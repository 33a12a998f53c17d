"""Loads ``_recognise`` (``csrc/recognise.cpp``): the plans of the usual kernels, found natively.

``plan(kernel)`` gives what ``tensor_ops.attention_plan`` or ``execute.fused_plan`` would, as a plain tuple, or None where
those have to look for themselves (and report what is wrong, if anything is): always where the extension is not built for this
interpreter, which costs time and nothing else.
"""
import importlib.machinery
import importlib.util
import pathlib

from . import ir, tensor_ops
from .affine import AffineMap

# (the first suffix names the interpreter's ABI: an extension built for another one is not found, and not loaded)
PATH = pathlib.Path(__file__).resolve().parent / "lib" / ("_recognise" + importlib.machinery.EXTENSION_SUFFIXES[0])


def _load():
    """The module's ``plan``, or a stand-in that knows no kernel."""
    if not PATH.exists():
        return lambda kernel: None
    loader = importlib.machinery.ExtensionFileLoader("_recognise", str(PATH))
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_recognise", loader))
    loader.exec_module(module)
    module.classes(ir.type, ir.value, AffineMap, ir.MemorySpace, ir.GemmWarpPolicy,
                   [ir.EndOp, ir.ParallelOp, ir.ForOp, ir.CopyOp, ir.FillOp, ir.ReduceOp, ir.GemmOp, tensor_ops.MmaOp,
                    tensor_ops.ReduceTensorOp, tensor_ops.LayoutViewOp, tensor_ops.TileStoreOp, tensor_ops.UpstreamOp])
    return module.plan


_plan = None


def plan(kernel):
    global _plan
    if kernel.__class__ is not ir.KernelOp:
        return None
    if _plan is None:
        _plan = _load()
    return _plan(kernel)
