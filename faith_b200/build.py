"""Builds faith_b200/libfaith_b200.so from csrc/ with nvcc for sm_100a (cross-compiles without a GPU), and the Python
boundary faith_b200/_binding.so from csrc/binding/ with the host compiler.

    python -m faith_b200.build            # incremental
    python -m faith_b200.build --force    # rebuild everything
"""
import concurrent.futures
import importlib.metadata
import os
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(CSRC, "build")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")
LIB = os.path.join(PKG, "libfaith_b200.so")
BINDING_SRC = os.path.join(CSRC, "binding", "binding.cpp")
BINDING = os.path.join(PKG, "_binding.so")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-I" + INCLUDE, "-I" + CSRC]


def _nvcc():
    cand = os.path.join(_cuda_home(), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cpp")))


def _newest_header():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return max(os.path.getmtime(h) for h in hs)


def _cuda_home():
    return os.environ.get("CUDA_HOME", "/usr/local/cuda")


def binding_target(torch_version=None):
    """What the extension module is built for: it uses torch's internal C++ interface, so another torch (or another
    interpreter) needs another build.  The module holds this text as `built_for`."""
    if torch_version is None:
        torch_version = importlib.metadata.version("torch")   # (without the import, which takes seconds)
    return "torch %s, %s" % (torch_version, sysconfig.get_config_var("SOABI"))


def _binding_current(path, target):
    newest = max(os.path.getmtime(BINDING_SRC), max(os.path.getmtime(os.path.join(INCLUDE, f)) for f in os.listdir(INCLUDE)))
    if not os.path.exists(path) or os.path.getmtime(path) < newest:
        return False
    with open(path, "rb") as f:
        return target.encode() + b"\0" in f.read()


def _build_binding(force, verbose):
    """The extension module that faith_b200/ops.py calls: host code only, linked against the C-ABI library next to it."""
    if not force and _binding_current(BINDING, binding_target()):
        return
    import torch
    troot = os.path.dirname(torch.__file__)
    tlib = os.path.join(troot, "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI),
           '-DFB_BUILT_FOR="%s"' % binding_target(torch.__version__),
           "-I" + INCLUDE, "-I" + os.path.join(troot, "include"),
           "-I" + os.path.join(troot, "include", "torch", "csrc", "api", "include"),
           "-I" + os.path.join(_cuda_home(), "include"), "-I" + sysconfig.get_paths()["include"],
           BINDING_SRC, "-o", BINDING, "-L" + PKG, "-lfaith_b200", "-L" + tlib, "-ltorch_python", "-ltorch_cpu", "-lc10",
           "-lc10_cuda", "-ltorch_cuda", "-L" + os.path.join(_cuda_home(), "lib64"), "-lcudart", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("building %s failed" % BINDING)


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    hdr = _newest_header()
    jobs = []
    objs = []
    for src in _sources():
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, os.path.splitext(src)[0] + ".o")
        objs.append(o)
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr):
            cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-x", "cu", "-c", s, "-o", o]
            jobs.append((src, cmd))

    def run(job):
        src, cmd = job
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r.returncode, r.stdout + r.stderr

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for src, rc, out in ex.map(run, jobs):
            if verbose or rc != 0:
                sys.stderr.write("[%s]\n%s\n" % (src, out))
            if rc != 0:
                raise RuntimeError("nvcc failed on %s" % src)
    if jobs or not os.path.exists(LIB):
        cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stdout + r.stderr)
    _build_binding(force, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
