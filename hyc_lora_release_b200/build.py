"""Build lib/libhyc.so (sm_100a) from csrc/*.cu with nvcc and the native host path lib/_hyc_host.so from csrc/host/*.cpp
with g++ against the installed torch.

    python hyc_lora_release_b200/build.py [--force] [-v]

Objects go to csrc/build/, the shared library to lib/.  Both are kept out of version
control; the libraries are what the Python layer loads (libhyc.so through ctypes, _hyc_host.so as an
extension module that links it).
"""
import concurrent.futures
import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(HERE, "lib", "libhyc.so")
HOST_LIB = os.path.join(HERE, "lib", "_hyc_host.so")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"] + os.environ.get("HYC_NVCC_EXTRA", "").split()


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found")
    return exe


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    os.makedirs(os.path.dirname(LIB), exist_ok=True)
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    nvcc = _nvcc()
    jobs = []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if force or _stale(obj, [src] + headers):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, r.stdout, r.stderr))
        return r.stderr

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        logs = list(ex.map(compile_one, jobs))
    if verbose:
        for log in logs:
            sys.stderr.write(log)
    objs = [os.path.join(OBJ, os.path.basename(s)[:-3] + ".o") for s in sources]
    if force or jobs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n%s\n%s" % (r.stdout, r.stderr))
    build_host(force)
    return LIB


def _torch_flags():
    """-> (compile flags, link flags) for code that includes torch/extension.h, from where the package is installed
    (importing torch only to ask it would cost the build most of its time)."""
    import importlib.util
    import sysconfig
    root = os.path.dirname(importlib.util.find_spec("torch").origin)
    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    cflags = ["-I" + os.path.join(root, "include"), "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
              "-isystem", cuda, "-I" + sysconfig.get_paths()["include"], "-DTORCH_EXTENSION_NAME=_hyc_host",
              "-DTORCH_API_INCLUDE_EXTENSION_H"]
    lib = os.path.join(root, "lib")
    return cflags, ["-L" + lib, "-Wl,-rpath," + lib, "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]


def build_host(force=False):
    sources = sorted(glob.glob(os.path.join(CSRC, "host", "*.cpp")))
    headers = glob.glob(os.path.join(CSRC, "host", "*.h")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    cflags, ldflags = _torch_flags()
    objs = {src: os.path.join(OBJ, os.path.basename(src)[:-4] + ".host.o") for src in sources}
    jobs = [(s, o) for s, o in objs.items() if force or _stale(o, [s] + headers)]

    def compile_one(job):
        src, obj = job
        r = subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-w"] + cflags + ["-c", src, "-o", obj],
                           capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("g++ failed for %s:\n%s\n%s" % (src, r.stdout, r.stderr))

    with concurrent.futures.ThreadPoolExecutor(max_workers=max(1, len(jobs))) as ex:
        list(ex.map(compile_one, jobs))
    if force or jobs or _stale(HOST_LIB, list(objs.values()) + [LIB]):
        cmd = ["g++", "-shared", "-o", HOST_LIB] + list(objs.values()) + ["-L" + os.path.dirname(LIB), "-l:libhyc.so", "-Wl,-rpath,$ORIGIN"] + ldflags
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n%s\n%s" % (r.stdout, r.stderr))
    return HOST_LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
