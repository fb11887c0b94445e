"""Native kernel build + load.

Parity: reference `colossalai/kernel/kernel_loader.py:31-131` + `extensions/{base,cpp,cuda}_extension.py`
(AOT/JIT build of op families, `KernelLoader.load()`).  B200-first differences:
  * ONE arch: every `.cu` is compiled with `-gencode arch=compute_100a,code=sm_100a -lineinfo`;
  * kernels export plain C launchers (`extern "C"`, raw pointers + cudaStream_t) and are loaded with ctypes, or called
    from one small torch module for the operators whose host time counts — no torch headers in the CUDA translation units, so a full rebuild takes seconds and the `.so` files live
    IN-TREE (`colossalai_b200/kernel/_build/`) so they travel to the GPU box with the repo snapshot;
  * on a GPU box a missing/unloadable library is a hard error (no silent eager fallback); on a CPU-only box the
    python ops use their torch reference path (the plumbing tier of the test-suite).
"""
from __future__ import annotations

import ctypes
import hashlib
import importlib.util
import os
import shutil
import subprocess
import sysconfig
import threading
import warnings
from pathlib import Path
from typing import Dict, List, Optional

import torch

__all__ = ["KernelLoader", "load", "build_all", "native_available", "launch_counter", "LIBS"]

_HERE = Path(__file__).resolve().parent
CSRC = _HERE / "csrc"
BUILD = _HERE / "_build"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--use_fast_math",
    "--expt-relaxed-constexpr", "--expt-extended-lambda", "-Xcompiler", "-fPIC", "-shared",
    "-U__CUDA_NO_HALF_OPERATORS__", "-U__CUDA_NO_HALF_CONVERSIONS__", "-U__CUDA_NO_BFLOAT16_CONVERSIONS__",
    "-U__CUDA_NO_HALF2_OPERATORS__",
]
CXX_FLAGS = ["-O3", "-std=c++17", "-fPIC", "-shared", "-fopenmp", "-ffast-math", "-fno-finite-math-only"]

# library name -> (sources, kind)
LIBS: Dict[str, dict] = {
    "cb200_elementwise": {"sources": ["elementwise.cu"], "kind": "cuda"},
    "cb200_norm": {"sources": ["norm.cu"], "kind": "cuda"},
    "cb200_optim": {"sources": ["multi_tensor_optim.cu"], "kind": "cuda"},
    "cb200_softmax": {"sources": ["softmax.cu"], "kind": "cuda"},
    "cb200_loss": {"sources": ["cross_entropy.cu"], "kind": "cuda"},
    "cb200_gemm": {"sources": ["gemm_tcgen05.cu"], "kind": "cuda"},
    "cb200_gemm_rows": {"sources": ["gemm_rows_tcgen05.cu"], "kind": "cuda"},
    "cb200_grouped_gemm": {"sources": ["grouped_gemm_tcgen05.cu"], "kind": "cuda"},
    "cb200_attn": {"sources": ["flash_attn_tcgen05.cu"], "kind": "cuda"},
    "cb200_comm": {"sources": ["fused_comm_gemm.cu"], "kind": "cuda"},
    "cb200_moe": {"sources": ["moe.cu"], "kind": "cuda"},
    "cb200_infer": {"sources": ["inference.cu"], "kind": "cuda"},
    "cb200_quant": {"sources": ["quant.cu"], "kind": "cuda"},
    # recurrences and softmax in IEEE fp32 (no approximate exp / division): built without --use_fast_math
    "cb200_mixers": {"sources": ["mixers.cu"], "kind": "cuda", "drop_flags": ["--use_fast_math"]},
    "cb200_cpu_adam": {"sources": ["cpu_adam.cpp"], "kind": "cpp"},
    "cb200_aio": {"sources": ["async_file_io.cpp"], "kind": "cpp", "extra": ["-lpthread"]},
    # the one library that sees torch: allocation, autograd and launches of the small hot operators (a python module)
    "cb200_host": {"sources": ["host_ops.cpp"], "kind": "torch"},
}


class _LaunchCounter:
    """Counts launches of OUR kernels (reported by bench.py as `gpu_launches`)."""

    def __init__(self) -> None:
        self._by_name: Dict[str, int] = {}
        self.enabled = True
        self.native = None              # counts of the launches that native code made since the last call

    def add(self, name: str, n: int = 1) -> None:
        if self.enabled:
            self._by_name[name] = self._by_name.get(name, 0) + n

    @property
    def by_name(self) -> Dict[str, int]:
        if self.native is not None:
            for name, n in self.native(True).items():
                self.add(name, n)
        return self._by_name

    @property
    def count(self) -> int:
        return sum(self.by_name.values())

    def reset(self) -> None:
        self.by_name.clear()


launch_counter = _LaunchCounter()
_loaded: Dict[str, ctypes.CDLL] = {}
_lock = threading.Lock()


def _nvcc() -> Optional[str]:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return cand if os.path.exists(cand) else None


def _src_hash(name: str) -> str:
    h = hashlib.sha1()
    spec = LIBS[name]
    for s in spec["sources"]:
        h.update((CSRC / s).read_bytes())
    for hdr in sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h")):
        h.update(hdr.read_bytes())
    h.update(" ".join(_flags(spec)).encode())
    if spec["kind"] == "torch":
        h.update(f"{torch.__version__} {sysconfig.get_config_var('EXT_SUFFIX')}".encode())
    return h.hexdigest()[:16]


def _flags(spec: dict) -> List[str]:
    if spec["kind"] == "torch":
        return ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]
    base = NVCC_FLAGS if spec["kind"] == "cuda" else CXX_FLAGS
    return [f for f in base if f not in spec.get("drop_flags", ())]


def lib_path(name: str) -> Path:
    return BUILD / f"lib{name}.so"


def is_stale(name: str) -> bool:
    p, stamp = lib_path(name), BUILD / f"{name}.hash"
    if not p.exists() or not stamp.exists():
        return True
    return stamp.read_text().strip() != _src_hash(name)


def build(name: str, verbose: bool = False, force: bool = False) -> Path:
    spec = LIBS[name]
    srcs = [str(CSRC / s) for s in spec["sources"]]
    for s in srcs:
        if not os.path.exists(s):
            raise FileNotFoundError(s)
    BUILD.mkdir(parents=True, exist_ok=True)
    out = lib_path(name)
    if not force and not is_stale(name):
        return out
    if spec["kind"] == "cuda":
        nvcc = _nvcc()
        if nvcc is None:
            raise RuntimeError("nvcc not found; cannot build CUDA kernels")
        cmd = [nvcc] + _flags(spec) + ["-I", str(CSRC)] + (["-Xptxas", "-v"] if verbose else []) + srcs + \
              ["-o", str(out), "-lcuda"] + spec.get("extra", [])
        # libcuda may be absent on the build box: resolve driver entry points at run time instead
        cmd = [c for c in cmd if c != "-lcuda"]
    elif spec["kind"] == "torch":
        root = Path(torch.__file__).resolve().parent
        cuda = Path(_nvcc() or "/usr/local/cuda/bin/nvcc").resolve().parent.parent
        inc = [root / "include", root / "include/torch/csrc/api/include", cuda / "include", sysconfig.get_paths()["include"]]
        cmd = ["g++"] + _flags(spec) + [f"-I{d}" for d in inc] + [f"-DTORCH_EXTENSION_NAME={name}", "-DTORCH_API_INCLUDE_EXTENSION_H",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + srcs + ["-o", str(out), f"-L{root / 'lib'}",
               "-lc10", "-ltorch_cpu", "-ltorch", "-ltorch_python", "-lc10_cuda", "-ltorch_cuda"]
    else:
        cmd = ["g++"] + _flags(spec) + ["-I", str(CSRC)] + srcs + ["-o", str(out)] + spec.get("extra", [])
    tmp = str(out) + f".tmp{os.getpid()}"
    cmd[cmd.index(str(out))] = tmp
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"build of {name} failed:\n{' '.join(cmd)}\n{res.stdout}\n{res.stderr}")
    os.replace(tmp, out)
    (BUILD / f"{name}.hash").write_text(_src_hash(name))
    if verbose:
        print(res.stderr)
    return out


def build_all(verbose: bool = False, force: bool = False, parallel: int = 8) -> List[Path]:
    from concurrent.futures import ThreadPoolExecutor

    names = [n for n, s in LIBS.items() if all((CSRC / x).exists() for x in s["sources"])]
    with ThreadPoolExecutor(max_workers=parallel) as ex:
        return list(ex.map(lambda n: build(n, verbose=verbose, force=force), names))


def native_available(name: str) -> bool:
    """True when the library can be used for CUDA tensors (GPU present and .so present/buildable)."""
    if LIBS[name]["kind"] != "cpp" and not torch.cuda.is_available():
        return False
    return lib_path(name).exists() or all((CSRC / s).exists() for s in LIBS[name]["sources"])


def load(name: str) -> ctypes.CDLL:
    with _lock:
        if name in _loaded:
            return _loaded[name]
        p = lib_path(name)
        if not p.exists() or (is_stale(name) and _nvcc() is not None and os.environ.get("CB200_NO_REBUILD") != "1"):
            try:
                build(name)
            except Exception:
                if not p.exists():
                    raise
        lib = ctypes.CDLL(str(p), mode=ctypes.RTLD_GLOBAL)
        _loaded[name] = lib
        return lib


# launchers that the host module calls, by library
_HOST_CALLS = {
    "cb200_norm": ["cb_rmsnorm_fwd", "cb_rmsnorm_bwd", "cb_norm_bwd_grid"],
    "cb200_moe": ["cb_moe_sort", "cb_moe_take_rows", "cb_moe_sum_rows", "cb_moe_sum_rows_bwd"],
    "cb200_grouped_gemm": ["cb_grouped_gemm", "cb_grouped_gemm_wgrad", "cb_grouped_gemm_gated", "cb_grouped_gemm_gated_bwd"],
    "cb200_elementwise": ["cb_glu_fwd_bounded", "cb_glu_bwd_bounded", "cb_rope", "cb_rope_pages"],
    "cb200_loss": ["cb_ce_row_stats", "cb_ce_loss_blocks", "cb_ce_loss", "cb_ce_softmax_grad"],
    "cb200_attn": ["cb_flash_attn_varlen_fwd", "cb_flash_attn_bwd"],
    "cb200_infer": ["cb_decode_num_splits", "cb_paged_decode_attention"],
    "cb200_gemm_rows": ["cb_gemm_rows", "cb_gemm_rows_gated", "cb_embed_rows"],
}
_host, _host_asked = None, False


def host():
    """The native host module (`csrc/host_ops.cpp`) with the kernels' launchers bound, or None where there is none for these
    sources and this torch: the python autograd functions launch the same kernels then."""
    global _host, _host_asked
    if not _host_asked:
        libs = {lib: load(lib) for lib in _HOST_CALLS}
        with _lock:
            if not _host_asked:
                _host = _load_host(libs)
                _host_asked = True
    return _host


def _load_host(libs):
    try:
        # bound to one torch and to the launchers' signatures: unlike a C library it is never taken as it was built for others
        if is_stale("cb200_host"):
            if os.environ.get("CB200_NO_REBUILD") == "1":
                raise RuntimeError("it was built for other sources or another torch, and CB200_NO_REBUILD=1")
            build("cb200_host")
        spec = importlib.util.spec_from_file_location("cb200_host", lib_path("cb200_host"))
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        mod.bind({f: ctypes.cast(getattr(libs[lib], f), ctypes.c_void_p).value for lib, fs in _HOST_CALLS.items() for f in fs})
    except Exception as e:
        warnings.warn(f"the native host module is not used, small operators run from python: {e}")
        return None
    launch_counter.native = mod.counts
    return mod


class KernelLoader:
    """Reference-style façade: `KernelLoader("cb200_norm").load()`."""

    def __init__(self, name: str) -> None:
        if name not in LIBS:
            raise KeyError(f"unknown kernel library {name!r}; known: {list(LIBS)}")
        self.name = name

    def is_available(self) -> bool:
        return native_available(self.name)

    def load(self) -> ctypes.CDLL:
        return load(self.name)


# --------------------------------------------------------------------------------------- ctypes helpers
def ptr(t: Optional[torch.Tensor]) -> ctypes.c_void_p:
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def stream_ptr() -> ctypes.c_void_p:
    return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(torch.cuda.current_device()))


WAIT_RAN_OUT = 702              # cudaErrorLaunchTimeout, as the attention launchers return it


def check(err: int, what: str) -> None:
    if err == WAIT_RAN_OUT:
        raise RuntimeError(f"{what}: a wait inside an earlier attention kernel ran out; what it wrote is not valid (CUDA error {err})")
    if err != 0:
        raise RuntimeError(f"{what}: native launcher returned CUDA error {err}")
