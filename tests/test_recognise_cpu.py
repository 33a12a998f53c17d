"""The native recogniser (csrc/recognise.cpp) against the Python ones: what it accepts they resolve to the same plan, also after
any single part of a built kernel has been changed, removed or put in another's place."""
import copy
import gc
import importlib
import os
import pickle
import random
import sysconfig
import tracemalloc

import pytest

import frisk_b200 as F
from frisk_b200 import build, capi, ir, recognise, tensor_ops

execute = importlib.import_module("frisk_b200.execute")
needs_build = pytest.mark.skipif(not recognise.PATH.exists(), reason="the native recogniser is not built")


def attention_kernel(n_q=64, n_kv=128, d=64, element="f16", out="f32", scale=0.125):
    s = F.create_session()
    ty = {"f16": s.builder.get_f16_ty, "bf16": s.builder.get_bf16_ty, "f32": s.builder.get_f32_ty}
    return F.build_attention_kernel(s.builder, s.module, "attention", n_q, n_kv, d, ty[element](), scale, ty[out]())


def gemm_kernel(m=48, n=32, k=64, dtype="fp16", fill=0.5, reduce="max", ta=False, tb=True, clear=False, out=None, trips=1):
    s = F.create_session()
    types = [s.memref_type(shape, t) for shape, t in
             (([k, m] if ta else [m, k], dtype), ([n, k] if tb else [k, n], dtype), ([m, n], out or dtype), ([m], out or dtype))]
    _, entry = s.new_kernel("fused", types)
    a, b, c, r = (entry.get_argument(i) for i in range(4))
    par = s.builder.create_parallel_op([4, 4], 128)
    s.builder.set_insertion_point_to_start(par.add_entry_block())

    def body(builder, iv):
        if fill is not None:
            builder.create_fill_op(c, fill, out or dtype)
        builder.create_gemm_op(a, b, c, ta, tb, clear)
        if reduce:
            builder.create_reduce_op(c, r, reduce, 1, True)
    s.builder.create_for_op(0, trips, 1, body)
    return s.module.get_kernel("fused")


def fields(desc):
    return [getattr(desc, name) for name, _ in desc._fields_]


def by_python(kernel):
    """What execute resolves the kernel to without the native recogniser; an exception counts as refused."""
    try:
        ops = tensor_ops._ops_of(kernel)
        if any(isinstance(op, tensor_ops.MmaOp) for op in ops):
            spec, idx = tensor_ops.attention_plan(kernel, ops)
            desc = capi.attn_desc(1, 1, spec["S_q"], spec["S_kv"], spec["D"], spec["scale"], False, spec["dtype_in"],
                                  spec["dtype_out"], normalize_p=True)
            return True, fields(desc), list(idx)
        desc, idx, epilogue = execute.fused_plan(kernel)
        return False, fields(desc), list(idx), epilogue
    except Exception:  # noqa: BLE001
        return None


def by_execute(kernel):
    attention, plan = execute._plan_of(kernel, capi.ALGO_AUTO)
    return (attention, fields(plan[0]), list(plan[1])) + (() if attention else (plan[2],))


KERNELS = {
    "attention": attention_kernel,
    "attention_bf16": lambda: attention_kernel(128, 64, 128, "bf16", "bf16", 0.5),
    "attention_bits": lambda: attention_kernel(scale=0x3E000000),
    "fused": gemm_kernel,
    "gemm": lambda: gemm_kernel(fill=None, reduce=None, ta=True, tb=False, clear=True),
    "fill": lambda: gemm_kernel(reduce=None, out="fp32"),
    "reduce": lambda: gemm_kernel(fill=None, reduce="add", clear=True, dtype="fp32"),
}


@needs_build
@pytest.mark.parametrize("name", KERNELS)
def test_usual_kernels_are_recognised(name):
    kernel = KERNELS[name]()
    assert recognise.plan(kernel) is not None
    assert by_execute(kernel) == by_python(kernel)


def parts_of(kernel):
    ops = [kernel] + tensor_ops._ops_of(kernel)
    values = [v for op in ops for v in op.operands + op.results] + list(kernel.regions[0].front().arguments)
    types = list({id(v.type): v.type for v in values}.values())
    return ops, values, types


def mutate(kernel, rng):
    """Changes one part of the kernel in place, the way a program that edits its IR might."""
    ops, values, types = parts_of(kernel)
    kind = rng.randrange(9)
    op = rng.choice(ops)
    odd = [0, 1, -1, 2, 3, 64, 128, 7, True, False, 0.0, -0.5, None, "max", "sum", "f16", [], [0], [1], (1.0, types[0])]
    if kind == 0 and op.attrs:
        op.attrs[rng.choice(sorted(op.attrs))] = rng.choice(odd)
    elif kind == 1 and op.attrs:
        del op.attrs[rng.choice(sorted(op.attrs))]
    elif kind == 2 and op.operands:
        op.operands[rng.randrange(len(op.operands))] = rng.choice(values)
    elif kind == 3 and op.operands:
        op.operands.pop(rng.randrange(len(op.operands)))
    elif kind == 4:
        rng.choice(values).type = rng.choice(types)
    elif kind == 5:
        t = rng.choice(types)
        choice = rng.randrange(4)
        if choice == 0:
            t.shape = rng.choice([[64, 64], [64], [64, 64, 1], (64, 128), [0, 64], [128, 64], [48, 32], [63, 64]])
        elif choice == 1:
            t.element = ir.type("float", name=rng.choice(["f16", "bf16", "f32", "f64"]))
        elif choice == 2:
            t.kind = rng.choice(["memref", "tensor", "float"])
        else:
            t.space = rng.choice(list(ir.MemorySpace))
    elif kind == 6:
        blk = rng.choice(ops[1:]).parent_block
        if blk is not None and len(blk.operations) > 1:
            moved = blk.operations.pop(rng.randrange(len(blk.operations)))
            if rng.random() < 0.7:
                blk.operations.insert(rng.randrange(len(blk.operations) + 1), moved)
    elif kind == 7:
        v = rng.choice(values)
        setattr(v, rng.choice(["index", "is_arg", "owner"]), rng.choice([0, 1, True, False, rng.choice(ops), values[0].owner]))
    else:
        op.op_name = rng.choice(["arith.mulf", "arith.divf", "arith.subf", "math.exp", "tensor.empty", "arith.truncf", "linalg.broadcast"])


@needs_build
@pytest.mark.parametrize("name", KERNELS)
def test_native_accepts_nothing_the_python_recognisers_refuse(name):
    accepted = 0
    for seed in range(1500):
        rng = random.Random(f"{name} {seed}")
        kernel = KERNELS[name]()
        for _ in range(rng.choice([1, 1, 2])):
            mutate(kernel, rng)
        if recognise.plan(kernel) is not None:
            accepted += 1
            assert by_execute(kernel) == by_python(kernel), seed
    assert accepted > 20  # (changes that leave the kernel what it was)


@needs_build
def test_unusual_kernels_are_left_to_python():
    class Mine(tensor_ops.MmaOp):
        pass
    kernel = attention_kernel()
    next(op for op in tensor_ops._ops_of(kernel) if isinstance(op, tensor_ops.MmaOp)).__class__ = Mine
    assert recognise.plan(kernel) is None and by_execute(kernel) == by_python(kernel)
    assert recognise.plan(gemm_kernel(fill=None, reduce=None, clear=True, trips=3)) is None
    assert recognise.plan(F.create_session().module) is None


def change_argument(kernel, index, shape):
    """Argument `index` and its views take another shape; the staging buffer and the ops on it stay as they are."""
    old = kernel.regions[0].front().arguments[index].type
    new = ir.type("memref", shape=list(shape), element=old.element, map=old.map, space=old.space)
    for v in parts_of(kernel)[1]:
        if v.type is old:
            v.type = new
    kernel.attrs["function_type"].inputs[index] = new
    return kernel


def store_through_buffer(shape, to_argument=False):
    """The result is stored to a staging buffer, which the output argument, of `shape`, was copied into (or is copied to)."""
    kernel = attention_kernel(64, 64, 64)
    store = next(op for op in tensor_ops._ops_of(kernel) if isinstance(op, tensor_ops.TileStoreOp))
    view = store.operands[1]
    buffer = tensor_ops.UpstreamOp("memref.alloc", (), [ir.type("memref", shape=[64, 64], element=view.type.element, map=None,
                                                                space=ir.MemorySpace.SHARED)])
    ends = [view, buffer.results[0]]
    copy = ir.CopyOp(operands=ends[::-1] if to_argument else ends, attrs={
        "srcMap": ir.AffineMap(empty=True), "dstMap": ir.AffineMap(empty=True), "srcExtents": [64, 64], "dstExtents": [64, 64], "_nsrc": 0})
    ops = store.parent_block.operations
    at = ops.index(store)
    ops[at:at + 1] = [buffer, store, copy] if to_argument else [buffer, copy, store]
    for op in (buffer, copy):
        op.parent_block = store.parent_block
    store.operands[1] = buffer.results[0]
    return change_argument(kernel, 3, shape)


@needs_build
@pytest.mark.parametrize("index,shape", [(0, [32, 64]), (1, [64, 64]), (2, [64, 64]), (1, [128, 32]), (2, [256, 32]), (0, [64, 128]), (1, [8192]),
                                         (1, [2, 64, 64])])
def test_an_argument_must_hold_the_tile_that_is_staged_from_it(index, shape):
    """The kernel would read the buffer's extents from the argument's address: beyond its end, or with another pitch."""
    kernel = change_argument(attention_kernel(64, 128, 64), index, shape)
    assert recognise.plan(kernel) is None
    with pytest.raises(ValueError, match="does not hold a tile"):
        execute._plan_of(kernel, capi.ALGO_AUTO)


@needs_build
@pytest.mark.parametrize("index,shape", [(0, [256, 64]), (1, [1, 128, 64]), (2, [129, 64]), (2, [3, 128, 64])])
def test_an_argument_may_hold_more_than_the_tile(index, shape):
    kernel = change_argument(attention_kernel(64, 128, 64), index, shape)
    plan = by_execute(kernel)
    assert plan == by_python(kernel) and plan[1:] == by_execute(attention_kernel(64, 128, 64))[1:]
    # but not where the copy names a place in it
    copy = [op for op in tensor_ops._ops_of(kernel) if isinstance(op, ir.CopyOp)][index]
    if shape[0] > 1:
        copy.attrs["srcMap"] = ir.AffineMap(num_dims=0, results=[ir.get_affine_constant_expr(64), ir.get_affine_constant_expr(0)])
        assert by_python(kernel) is None and recognise.plan(kernel) is None


@needs_build
@pytest.mark.parametrize("shape", [[32, 64], [64, 64]])
@pytest.mark.parametrize("to_argument", [False, True])
def test_a_result_is_stored_to_an_argument(shape, to_argument):
    """A buffer that an argument was copied into is not that argument."""
    kernel = store_through_buffer(shape, to_argument)
    assert recognise.plan(kernel) is None
    with pytest.raises(ValueError, match="global kernel arguments"):
        execute._plan_of(kernel, capi.ALGO_AUTO)


@pytest.mark.parametrize("name", ["attention", "fused"])
def test_entry_arguments_are_those_of_the_function_type(name):
    """The tensors are checked against the function type, and the plan comes from the entry block's arguments: both must agree."""
    import torch
    kernel = KERNELS[name]()
    inputs = kernel.attrs["function_type"].inputs
    dtypes = {"f16": torch.float16, "f32": torch.float32}

    def run():
        execute.execute(kernel, *[torch.zeros(t.shape, dtype=dtypes[t.element.name]) for t in inputs])
    inputs[0] = ir.type("memref", shape=list(inputs[0].shape), element=inputs[0].element, map=inputs[0].map, space=inputs[0].space)
    with pytest.raises(ValueError, match="no CPU path"):  # (equal types; the tensors are not on a GPU)
        run()
    assert recognise.plan(kernel) is None  # (left to Python, which compares them)
    inputs[0].shape = [16, 64]
    with pytest.raises(ValueError, match="entry block"):
        run()
    inputs.append(inputs[1])
    with pytest.raises(ValueError, match="entry block"):
        run()


@pytest.mark.parametrize("name", KERNELS)
def test_plans_are_the_same_without_the_extension(name, monkeypatch, tmp_path):
    monkeypatch.setattr(recognise, "PATH", tmp_path / "_recognise.so")
    monkeypatch.setattr(recognise, "_plan", None)
    kernel = KERNELS[name]()
    assert recognise.plan(kernel) is None and by_execute(kernel) == by_python(kernel)


def test_the_extension_is_built_for_this_interpreter_or_not_at_all(monkeypatch, tmp_path, capsys):
    assert recognise.PATH.name == "_recognise" + sysconfig.get_config_var("EXT_SUFFIX") and build.RECOGNISE == recognise.PATH
    target = tmp_path / recognise.PATH.name
    monkeypatch.setattr(build, "RECOGNISE", target)
    with monkeypatch.context() as m:
        m.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})  # no Python.h there
        assert build.build_recognise() is None and "without the native recogniser" in capsys.readouterr().err
    target.write_bytes(b"of an older source")
    os.utime(target, (0, 0))
    monkeypatch.setattr(build.shutil, "which", lambda name: None)  # no g++
    assert build.build_recognise() is None and not target.exists()


@needs_build
@pytest.mark.parametrize("make", [attention_kernel, gemm_kernel])
def test_recognising_leaves_nothing_in_the_kernel(make):
    """A kernel's objects hold no more memory after a call than before (an instance dictionary is made when somebody asks for it)."""
    assert recognise.plan(make()) is not None  # (sets up what a process keeps)
    kernel = make()
    gc.collect()
    tracemalloc.start()
    try:
        recognise.plan(kernel)
        assert tracemalloc.get_traced_memory()[0] < 200  # (the interpreter's own; a dictionary takes 100 and more, and there are dozens)
    finally:
        tracemalloc.stop()


@pytest.mark.parametrize("protocol", range(pickle.HIGHEST_PROTOCOL + 1))
def test_kernels_are_saved_and_copied_whole(protocol):
    kernel = gemm_kernel()
    kernel.note = "kept"
    for other in (pickle.loads(pickle.dumps(kernel, protocol)), copy.deepcopy(kernel)):
        assert str(other) == str(kernel) and other.note == "kept" and by_python(other) == by_python(kernel) is not None
    v = kernel.regions[0].blocks[0].arguments[1]
    old = ir.value.__new__(ir.value)
    old.__setstate__({"type": v.type, "owner": v.owner, "index": 1, "is_arg": True})  # as it was saved without slots
    assert (old.type, old.owner, old.index, old.is_arg) == (v.type, v.owner, 1, True)
