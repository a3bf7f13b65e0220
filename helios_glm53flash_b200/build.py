"""Builds libhelios_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU)."""
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libhelios_b200.so")
BINDING = os.path.join(HERE, "_binding.so")
SOURCES = [
    "status.cu", "kda_conv.cu", "kda_glue.cu", "kda_recurrent.cu", "kda_chunked.cu", "indexer_aux.cu",
    "indexer_score.cu", "dsa_topk.cu", "mla_attend.cu", "mla_flash_tc.cu", "mla_append.cu", "absorb.cu", "absorb_tc.cu",
    "tc05_selftest.cu", "shim.cu",
]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--use_fast_math", "-Xcompiler", "-fPIC,-fvisibility=hidden", "-Xptxas", "-v",
]


def _newer(src, dst):
    if not os.path.exists(dst):
        return True
    t = os.path.getmtime(dst)
    deps = [src] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".hpp"))]
    deps += [os.path.join(HERE, "..", "include", f) for f in os.listdir(os.path.join(HERE, "..", "include"))]
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(name, verbose):
    src = os.path.join(CSRC, name)
    obj = os.path.join(OBJ, name.replace(".cu", ".o"))
    if not _newer(src, obj):
        return obj, ""
    cmd = ["nvcc"] + NVCC_FLAGS + ["-c", src, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s" % (name, r.stderr))
    return obj, r.stderr if verbose else ""


def _build_binding():
    """The CPython call path (csrc/binding.cpp): host code against torch's headers; the torch libraries it names are the ones
    that `import torch` has loaded already."""
    src = os.path.join(CSRC, "binding.cpp")
    if not _newer(src, BINDING):
        return
    import sysconfig
    from importlib.util import find_spec
    torch_dir = os.path.dirname(find_spec("torch").origin)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    inc = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-w", src, "-o", BINDING + ".tmp"]
    cmd += ["-I" + d for d in inc] + ["-L" + os.path.join(torch_dir, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed for binding.cpp:\n" + r.stderr)
    os.replace(BINDING + ".tmp", BINDING)


def build(verbose=False, force=False):
    """Compile every CUDA source and link the shared library, and the Python binding beside it; returns the library's path."""
    os.makedirs(OBJ, exist_ok=True)
    if force:
        for f in os.listdir(OBJ):
            os.remove(os.path.join(OBJ, f))
        if os.path.exists(BINDING):
            os.remove(BINDING)
    with ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as ex:
        binding = ex.submit(_build_binding)
        results = list(ex.map(lambda n: _compile(n, verbose), SOURCES))
        binding.result()
    objs = [o for o, _ in results]
    if verbose:
        for _, log in results:
            if log:
                sys.stderr.write(log)
    if (not os.path.exists(LIB)) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        cmd = ["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", LIB] + objs
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stderr)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
