"""Build recipe of the product library `libaotx_q8_b200.so` (hand-written CUDA for sm_100a).

The library is built in-tree with nvcc; nothing is compiled at import time.  `build()`
rebuilds only the objects whose sources changed.
"""
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libaotx_q8_b200.so")
# The Python module of csrc/host_calls.c, under the name that only the interpreter it is built for looks for.
CALLS = os.path.join(HERE, "_host_calls" + sysconfig.get_config_var("EXT_SUFFIX"))
SOURCES = ["q8_api.cu", "q8_simt.cu", "q8_dispatch.cu", "q8_stream.cu", "q8_decode.cu", "q8_decode_warp.cu", "q8_decode_rows.cu", "q8_mid.cu", "q8_pair.cu", "q8_wide.cu", "q8_static.cu", "q8_moe.cu", "q8_route.cu", "q8_peers.cu",
           "q_generic.cu", "q_warp.cu", "gguf_table.cpp", "gguf_upload.cu"]
HEADERS = ["q8_common.cuh", "q8_ptx.cuh", "q8_warp_ptx.cuh", "q8_rows.cuh", "q8_schedule.cuh", "q8_decode_operands.cuh", "q8_store.cuh", "q8_simt_gemv.cuh", "q8_route.cuh", "q8_launch.h", "q8_tile.cuh", "q_blocks.cuh", os.path.join("..", "..", "include", "aotx_q8_b200.h"),
           os.path.join("..", "..", "include", "aotx_gguf_b200.h")]
NVCC_FLAGS = ["-std=c++17", "-O3", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a",
              "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    stamp = os.path.getmtime(target)
    return any(os.path.getmtime(d) > stamp for d in deps)


def _compile(src):
    obj = os.path.join(OBJ, os.path.splitext(src)[0] + ".o")
    deps = [os.path.join(CSRC, src)] + [os.path.join(CSRC, h) for h in HEADERS]
    log = obj + ".ptxas.log"   # what ptxas -v said for this object: registers, spills, shared memory
    if not _stale(obj, deps) and os.path.exists(log):
        return obj, ""
    cmd = ["nvcc", *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s" % (src, done.stderr))
    with open(log, "w") as f:
        f.write(done.stderr)
    return obj, done.stderr


def resource_usage():
    """{kernel or out-of-line function (mangled): {"registers": r (kernels only), "spill_stores": s,
    "spill_loads": l, "stack": b}} from the ptxas reports kept beside the objects (build() first)."""
    import re
    usage = {}
    for src in SOURCES:
        log = os.path.join(OBJ, os.path.splitext(src)[0] + ".o.ptxas.log")
        if not os.path.exists(log):
            continue
        name = None      # the kernel that is being compiled
        about = None     # the function that the next frame and spills belong to
        for line in open(log):
            found = re.search(r"Compiling entry function '([^']+)'", line)
            if found:
                name = found.group(1)
                usage[name] = {}
                continue
            found = re.search(r"Function properties for (\S+)", line)
            if found:
                about = found.group(1)
                continue
            found = re.search(r"(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", line)
            if found and about is not None:
                usage.setdefault(about, {}).update(stack=int(found.group(1)), spill_stores=int(found.group(2)),
                                                   spill_loads=int(found.group(3)))
            found = re.search(r"Used (\d+) registers", line)
            if found and name is not None:
                usage[name]["registers"] = int(found.group(1))
    return usage


def _build_calls(include=sysconfig.get_paths()["include"]):
    """The module of csrc/host_calls.c.  Only Python programs are faster with it, and without it they call through
    ctypes: where there are no Python headers or no gcc, the library is all that is built."""
    calls = os.path.join(CSRC, "host_calls.c")
    if not os.path.exists(os.path.join(include, "Python.h")) or shutil.which("gcc") is None:
        print("no Python headers or no gcc: " + os.path.basename(CALLS) + " is not built", file=sys.stderr)
        return
    if _stale(CALLS, [calls, os.path.join(CSRC, "..", "..", "include", "aotx_q8_b200.h")]):
        subprocess.run(["gcc", "-O2", "-Wall", "-Werror", "-shared", "-fPIC", "-I" + include, "-o", CALLS, calls], check=True)


def build(verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    with ThreadPoolExecutor(max_workers=len(SOURCES)) as pool:
        results = list(pool.map(_compile, SOURCES))
    objs = [r[0] for r in results]
    log = "".join(r[1] for r in results)
    if log:
        with open(os.path.join(OBJ, "ptxas.log"), "w") as f:
            f.write(log)
    if _stale(LIB, objs):
        subprocess.run(["nvcc", "-shared", "-o", LIB, *objs, "-gencode",
                        "arch=compute_100a,code=sm_100a"], check=True)
    _build_calls()
    untagged = os.path.join(HERE, "_host_calls.so")     # of a build before the name said so; any interpreter would load it
    if os.path.exists(untagged):
        os.remove(untagged)
    if verbose and log:
        print(log)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
