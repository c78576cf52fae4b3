"""Builds ``csrc/liboeq_b200.so`` in-tree with nvcc for sm_100a.

Usage: ``python -m openequivariance_b200.build_native [--force]``.  The kernel templates under
``csrc/kernels/`` are embedded into the library as raw string literals (``kernels_embed.inc``, generated
here) because they are specialised per problem at run time by NVRTC; the few problem-independent kernels
are compiled ahead of time by nvcc with the rest of the host code.
"""

from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(CSRC, "liboeq_b200.so")
STAMP = LIB + ".srchash"
EMBED = {"K_COMMON": "common.cuh", "K_GENERIC": "generic_tp.cuh", "K_DW_REDUCE": "dw_reduce.cuh", "K_FAST_UVU": "fast_uvu.cuh",
         "K_UVW_TC": "uvw_tc.cuh", "K_UVW_ITEM": "uvw_item.cuh", "K_UVW_F64": "uvw_f64.cuh", "K_SYM_POLY": "sym_poly.cuh"}


def _sources():
    out = [os.path.join(CSRC, "oeq_b200.cu"), os.path.join(CSRC, "dealing.h"), os.path.join(CSRC, "graph_prep.cuh"), os.path.join(CSRC, "group_mm.cuh"),
           os.path.join(CSRC, "sym_contraction.cuh"), os.path.join(CSRC, "partition_plan.cuh"),
           os.path.join(HERE, "..", "include", "oeq_b200.h")]
    out += [os.path.join(CSRC, "kernels", f) for f in EMBED.values()]
    return [p for p in out if os.path.exists(p)]


def write_embed() -> str:
    path = os.path.join(CSRC, "kernels_embed.inc")
    parts = ["// generated by build_native.py from csrc/kernels/*.cuh -- do not edit\n"]
    for name, fname in EMBED.items():
        fpath = os.path.join(CSRC, "kernels", fname)
        text = open(fpath).read() if os.path.exists(fpath) else ""
        assert ')OEQK"' not in text
        # split into chunks: some compilers cap the length of a single string literal
        chunks = [text[i:i + 12000] for i in range(0, len(text), 12000)] or [""]
        body = "\n".join(f'R"OEQK({c})OEQK"' for c in chunks)
        parts.append(f"static const char {name}[] =\n{body};\n")
    new = "".join(parts)
    if not os.path.exists(path) or open(path).read() != new:
        with open(path, "w") as f:
            f.write(new)
    return path


def _source_hash() -> str:
    import hashlib
    h = hashlib.sha256()
    for p in sorted(_sources()):
        h.update(os.path.basename(p).encode())
        h.update(open(p, "rb").read())
    return h.hexdigest()


def needs_build() -> bool:
    """True when the library is missing or was built from other sources (a content hash, kept beside the
    library, decides: file times do not survive a copy to another machine)."""
    if not os.path.exists(LIB) or not os.path.exists(STAMP):
        return True
    return open(STAMP).read().strip() != _source_hash()


def build(force: bool = False, verbose: bool = True) -> str:
    if not force and not needs_build():
        return LIB
    write_embed()
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O2", "-std=c++17", "-shared",
           "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "-o", LIB + f".tmp{os.getpid()}",
           os.path.join(CSRC, "oeq_b200.cu"),
           "-L/usr/local/cuda/lib64", "-lnvrtc", "-ldl", "-Xlinker", "-rpath=/usr/local/cuda/lib64"]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    os.replace(LIB + f".tmp{os.getpid()}", LIB)   # another process may be loading the old file right now
    with open(STAMP + f".tmp{os.getpid()}", "w") as f:
        f.write(_source_hash())
    os.replace(STAMP + f".tmp{os.getpid()}", STAMP)
    return LIB


# ---- the torch operator library (C++ registration of the libtorch_tp_jit ops) ----------------------------------
TORCH_LIB = os.path.join(CSRC, "liboeq_b200_torch.so")
TORCH_STAMP = TORCH_LIB + ".srchash"
TORCH_SRC = os.path.join(CSRC, "torch_ops.cpp")


def _torch_source_hash() -> str:
    import hashlib

    import torch
    h = hashlib.sha256()
    h.update(torch.__version__.encode())
    for p in (TORCH_SRC, os.path.join(HERE, "..", "include", "oeq_b200.h")):
        h.update(open(p, "rb").read())
    return h.hexdigest()


def torch_ops_need_build() -> bool:
    if not os.path.exists(TORCH_LIB) or not os.path.exists(TORCH_STAMP):
        return True
    return open(TORCH_STAMP).read().strip() != _torch_source_hash()


def build_torch_ops(force: bool = False, verbose: bool = True) -> str:
    """Compiles ``csrc/torch_ops.cpp`` against the installed torch into ``csrc/liboeq_b200_torch.so`` (in-tree, beside
    ``liboeq_b200.so``, which it links).  Needs g++ and torch's headers; no GPU."""
    if not force and not torch_ops_need_build():
        return TORCH_LIB
    build(force=False, verbose=verbose)
    import torch
    from torch.utils import cpp_extension as ce
    torch_lib = ce.library_paths()[0]
    cxx = os.environ.get("CXX", "g++")
    tmp = TORCH_LIB + f".tmp{os.getpid()}"
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-o", tmp, TORCH_SRC,
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += [f"-I{p}" for p in ce.include_paths()] + ["-I/usr/local/cuda/include"]
    cmd += [f"-L{torch_lib}", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", f"-L{CSRC}", "-loeq_b200",
            "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{torch_lib}"]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    os.replace(tmp, TORCH_LIB)
    with open(TORCH_STAMP + f".tmp{os.getpid()}", "w") as f:
        f.write(_torch_source_hash())
    os.replace(TORCH_STAMP + f".tmp{os.getpid()}", TORCH_STAMP)
    return TORCH_LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv)
    print(LIB)
    if "--torch" in sys.argv:
        print(build_torch_ops(force="--force" in sys.argv))
