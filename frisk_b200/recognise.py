"""Loads ``_recognise`` (``csrc/recognise.cpp``): the plans of the usual kernels, found natively.

``plan(kernel)`` gives what ``tensor_ops.attention_plan`` or ``execute.fused_plan`` would, as a plain tuple, or None where
those have to look for themselves (and report what is wrong, if anything is).
"""
import importlib.machinery
import importlib.util
import pathlib

from . import ir, tensor_ops
from .affine import AffineMap

PATH = pathlib.Path(__file__).resolve().parent / "lib" / "_recognise.so"


def _load():
    if not PATH.exists():
        raise RuntimeError(f"{PATH} is missing: build it with `python -m frisk_b200.build`")
    loader = importlib.machinery.ExtensionFileLoader("_recognise", str(PATH))
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_recognise", loader))
    loader.exec_module(module)
    module.classes(ir.type, ir.value, AffineMap, ir.MemorySpace, ir.GemmWarpPolicy,
                   [ir.EndOp, ir.ParallelOp, ir.ForOp, ir.CopyOp, ir.FillOp, ir.ReduceOp, ir.GemmOp, tensor_ops.MmaOp,
                    tensor_ops.ReduceTensorOp, tensor_ops.LayoutViewOp, tensor_ops.TileStoreOp, tensor_ops.UpstreamOp])
    return module


_module = None


def plan(kernel):
    global _module
    if kernel.__class__ is not ir.KernelOp:
        return None
    if _module is None:
        _module = _load()
    return _module.plan(kernel)
