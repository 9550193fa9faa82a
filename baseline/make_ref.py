"""Build ``baseline/_ref/`` — an importable copy of the UNMODIFIED reference package.

The reference tree does not install (`pip install /root/reference` -> "Neither 'setup.py' nor
'pyproject.toml' found") and does not import as shipped: ``deepspeed/accelerator``,
``deepspeed/ops/op_builder`` and ``deepspeed/ops/csrc`` are 10-16 byte text files (dangling symlink
stubs), so ``import deepspeed`` dies with ``No module named 'deepspeed.accelerator'``.

This script copies every reference file byte-for-byte and puts two tiny *additional* packages where
the three stubs are:

* ``deepspeed/accelerator``      a CUDA-only ``get_accelerator()`` exposing the methods the reference calls;
* ``deepspeed/ops/op_builder``   builder classes that exist but report ``is_compatible() == False`` (their
  native sources are absent from the reference) — the benchmark config uses ``torch_adam: true`` so no
  builder is ever loaded.

Nothing of this repository's engine, kernels or models is on the reference path.
"""
import os
import shutil
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = "/root/reference/deepspeed"
DST = os.path.join(HERE, "_ref", "deepspeed")

ACCELERATOR = r'''
"""CUDA-only accelerator shim (generated by baseline/make_ref.py; not part of the reference)."""
import functools
import os
import torch


class CUDA_Accelerator:
    _name = "cuda"
    _communication_backend_name = "nccl"
    _compile_backend = "inductor"

    def is_synchronized_device(self): return False
    def use_host_timers(self): return self.is_synchronized_device()
    def resolves_data_dependency(self): return self.is_synchronized_device()
    def handles_memory_backpressure(self): return self.is_synchronized_device()
    def device_name(self, device_index=None): return "cuda" if device_index is None else f"cuda:{device_index}"
    def device(self, device_index=None): return torch.cuda.device(device_index)
    def set_device(self, device_index): torch.cuda.set_device(device_index)
    def current_device(self): return torch.cuda.current_device()
    def current_device_name(self): return f"cuda:{torch.cuda.current_device()}"
    def device_count(self): return torch.cuda.device_count()
    def synchronize(self, device_index=None): return torch.cuda.synchronize(device_index)
    def random(self): return torch.random
    def set_rng_state(self, new_state, device_index=None):
        return torch.cuda.set_rng_state(new_state) if device_index is None else torch.cuda.set_rng_state(new_state, device_index)
    def get_rng_state(self, device_index=None):
        return torch.cuda.get_rng_state() if device_index is None else torch.cuda.get_rng_state(device_index)
    def manual_seed(self, seed): return torch.cuda.manual_seed(seed)
    def manual_seed_all(self, seed): return torch.cuda.manual_seed_all(seed)
    def initial_seed(self): return torch.cuda.initial_seed()
    def default_generator(self, device_index): return torch.cuda.default_generators[device_index]
    @property
    def Stream(self): return torch.cuda.Stream
    def stream(self, stream): return torch.cuda.stream(stream)
    def current_stream(self, device_index=None): return torch.cuda.current_stream(device_index)
    def default_stream(self, device_index=None): return torch.cuda.default_stream(device_index)
    @property
    def Event(self): return torch.cuda.Event
    def empty_cache(self): return torch.cuda.empty_cache()
    def memory_allocated(self, device_index=None): return torch.cuda.memory_allocated(device_index)
    def max_memory_allocated(self, device_index=None): return torch.cuda.max_memory_allocated(device_index)
    def reset_max_memory_allocated(self, device_index=None): return torch.cuda.reset_peak_memory_stats(device_index)
    def memory_cached(self, device_index=None): return torch.cuda.memory_reserved(device_index)
    def max_memory_cached(self, device_index=None): return torch.cuda.max_memory_reserved(device_index)
    def reset_max_memory_cached(self, device_index=None): return torch.cuda.reset_peak_memory_stats(device_index)
    def memory_stats(self, device_index=None): return torch.cuda.memory_stats(device_index)
    def reset_peak_memory_stats(self, device_index=None): return torch.cuda.reset_peak_memory_stats(device_index)
    def memory_reserved(self, device_index=None): return torch.cuda.memory_reserved(device_index)
    def max_memory_reserved(self, device_index=None): return torch.cuda.max_memory_reserved(device_index)
    def total_memory(self, device_index=None): return torch.cuda.get_device_properties(device_index or 0).total_memory
    def available_memory(self, device_index=None): return torch.cuda.mem_get_info(device_index)[0]
    def is_bf16_supported(self): return True
    def is_fp16_supported(self): return True
    def supported_dtypes(self): return [torch.float, torch.half, torch.bfloat16]
    def is_triton_supported(self): return False
    def amp(self): return torch.cuda.amp
    def is_available(self): return torch.cuda.is_available()
    def range_push(self, msg): return torch.cuda.nvtx.range_push(msg)
    def range_pop(self): return torch.cuda.nvtx.range_pop()
    def lazy_call(self, callback): return torch.cuda._lazy_call(callback)
    def communication_backend_name(self): return self._communication_backend_name
    def communication_backend_version(self): return torch.cuda.nccl.version()
    def create_graph(self): return torch.cuda.CUDAGraph()
    def capture_to_graph(self, graph, pool=None, stream=None): return torch.cuda.graph(graph, pool, stream)
    def replay_graph(self, graph): graph.replay()
    @property
    def BFloat16Tensor(self): return functools.partial(torch.tensor, dtype=torch.bfloat16, device="cuda")
    @property
    def ByteTensor(self): return functools.partial(torch.tensor, dtype=torch.uint8, device="cuda")
    @property
    def DoubleTensor(self): return functools.partial(torch.tensor, dtype=torch.double, device="cuda")
    @property
    def FloatTensor(self): return functools.partial(torch.tensor, dtype=torch.float, device="cuda")
    @property
    def HalfTensor(self): return functools.partial(torch.tensor, dtype=torch.half, device="cuda")
    @property
    def IntTensor(self): return functools.partial(torch.tensor, dtype=torch.int, device="cuda")
    @property
    def LongTensor(self): return functools.partial(torch.tensor, dtype=torch.long, device="cuda")
    def pin_memory(self, tensor, align_bytes=1): return tensor.pin_memory()
    def is_pinned(self, tensor): return tensor.is_pinned()
    def on_accelerator(self, tensor): return str(tensor.device).startswith("cuda:")
    def op_builder_dir(self): return "deepspeed.ops.op_builder"
    def create_op_builder(self, class_name):
        import deepspeed.ops.op_builder as ob
        return getattr(ob, class_name)()
    def get_op_builder(self, class_name):
        import deepspeed.ops.op_builder as ob
        return getattr(ob, class_name)
    def build_extension(self):
        from torch.utils.cpp_extension import BuildExtension
        return BuildExtension
    def export_envs(self): return ["NCCL"]
    def visible_devices_envs(self): return ["CUDA_VISIBLE_DEVICES"]
    def set_visible_devices_envs(self, current_env, local_accelerator_ids):
        for env in self.visible_devices_envs():
            current_env[env] = ",".join(map(str, local_accelerator_ids))
    def get_compile_backend(self): return self._compile_backend
    def set_compile_backend(self, backend): self._compile_backend = backend
    def is_fp(self, dtype): return dtype in (torch.float, torch.half, torch.bfloat16)


_ACC = None


def get_accelerator():
    global _ACC
    if _ACC is None:
        _ACC = CUDA_Accelerator()
    return _ACC


def set_accelerator(accel_obj):
    global _ACC
    _ACC = accel_obj


def is_current_accelerator_supported():
    return True
'''

ACCELERATOR_REAL = '''
from .real_accelerator import get_accelerator, set_accelerator, is_current_accelerator_supported
'''

OP_BUILDER = r'''
"""op_builder shim (generated by baseline/make_ref.py): the reference's native sources (csrc/) are absent,
so every builder exists, reports itself incompatible and refuses to load."""


class OpBuilder:
    NAME = "deepspeed_not_implemented"
    BUILD_VAR = "DS_BUILD_NONE"

    def __init__(self, name=None):
        self.name = name or self.NAME

    def absolute_name(self):
        return f"deepspeed.ops.{self.NAME}_op"

    def is_compatible(self, verbose=False):
        return False

    def load(self, verbose=True):
        raise RuntimeError(f"{type(self).__name__}: native op sources are not part of the reference tree")

    def sources(self): return []
    def include_paths(self): return []
    def extra_ldflags(self): return []
    def compute_capability_args(self, cross_compile_archs=None): return []
    def builder(self): raise RuntimeError("no native sources")
    def installed_cuda_version(self, name=""): return (0, 0)


class NotImplementedBuilder(OpBuilder):
    pass


_NAMES = ["AsyncIOBuilder", "GDSBuilder", "CPUAdamBuilder", "CPUAdagradBuilder", "CPULionBuilder", "FusedAdamBuilder",
          "FusedLambBuilder", "FusedLionBuilder", "QuantizerBuilder", "FPQuantizerBuilder", "TransformerBuilder",
          "StochasticTransformerBuilder", "InferenceBuilder", "SpatialInferenceBuilder", "InferenceCoreBuilder",
          "InferenceCutlassBuilder", "RaggedOpsBuilder", "RaggedUtilsBuilder", "RandomLTDBuilder", "EvoformerAttnBuilder",
          "UtilsBuilder", "PackbitsBuilder", "SparseAttnBuilder", "ShareMemCommBuilder", "CCLCommBuilder",
          "DeepCompileBuilder"]
for _n in _NAMES:
    globals()[_n] = type(_n, (OpBuilder,), {"NAME": _n.replace("Builder", "").lower()})


def get_default_compute_capabilities():
    return "10.0"


def __getattr__(name):
    if name.endswith("Builder"):
        cls = type(name, (OpBuilder,), {"NAME": name.replace("Builder", "").lower()})
        globals()[name] = cls
        return cls
    raise AttributeError(name)
'''


def is_staged(dst=None):
    """True when the staged copy is complete (package file + both shim packages present)."""
    dst = dst or DST
    return all(os.path.isfile(os.path.join(dst, *p)) for p in (
        ("__init__.py",), ("runtime", "engine.py"), ("accelerator", "real_accelerator.py"),
        ("ops", "op_builder", "all_ops.py")))


def main():
    if not os.path.isdir(SRC):
        raise FileNotFoundError(
            f"{SRC} does not exist on this machine: stage the reference where it is mounted by running "
            f"`python __graft_entry__.py` (build() calls baseline/make_ref.py); baseline/_ref then ships with the tree")
    if os.path.isdir(DST):
        shutil.rmtree(DST)
    os.makedirs(os.path.dirname(DST), exist_ok=True)

    def ignore(d, names):
        return [n for n in names if n == "__pycache__"]

    shutil.copytree(SRC, DST, ignore=ignore, copy_function=shutil.copyfile)
    for stub in ("accelerator", os.path.join("ops", "op_builder"), os.path.join("ops", "csrc")):
        p = os.path.join(DST, stub)
        if os.path.isfile(p):
            os.chmod(p, 0o644)
            os.remove(p)
        os.makedirs(p, exist_ok=True)
    for dp, _, fns in os.walk(DST):
        os.chmod(dp, 0o755)
        for fn in fns:
            os.chmod(os.path.join(dp, fn), 0o644)
    acc = os.path.join(DST, "accelerator")
    open(os.path.join(acc, "real_accelerator.py"), "w").write(ACCELERATOR)
    open(os.path.join(acc, "__init__.py"), "w").write(ACCELERATOR_REAL)
    open(os.path.join(acc, "abstract_accelerator.py"), "w").write("class DeepSpeedAccelerator:\n    pass\n")
    open(os.path.join(acc, "cuda_accelerator.py"), "w").write("from .real_accelerator import CUDA_Accelerator\n")
    ob = os.path.join(DST, "ops", "op_builder")
    open(os.path.join(ob, "__init__.py"), "w").write(OP_BUILDER)
    open(os.path.join(ob, "builder.py"), "w").write("from . import OpBuilder, get_default_compute_capabilities\n")
    open(os.path.join(ob, "all_ops.py"), "w").write(
        "from . import _NAMES\nfrom . import *  # noqa\nimport deepspeed.ops.op_builder as _ob\n"
        "__op_builders__ = [getattr(_ob, n)() for n in _NAMES]\n"
        "ALL_OPS = {b.NAME: b for b in __op_builders__}\naccelerator_name = 'cuda'\n")
    open(os.path.join(ob, "dc.py"), "w").write("from . import DeepCompileBuilder\n")
    open(os.path.join(ob, "async_io.py"), "w").write("from . import AsyncIOBuilder\n")
    open(os.path.join(DST, "ops", "csrc", "README"), "w").write("native sources are absent from the reference tree\n")
    print("reference package staged at", DST)


if __name__ == "__main__":
    main()
