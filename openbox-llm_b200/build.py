"""Build libnsa_b200.so (the C-ABI library) in-tree with nvcc for sm_100a, and _nsa_torch.so, the autograd nodes on top
of it, with the host compiler against the installed torch."""
import hashlib
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(CSRC, "libnsa_b200.so")
EXT = os.path.join(CSRC, "_nsa_torch.so")
SOURCES = ["api.cu", "simt.cu", "simt_tile.cu", "f32_tile.cu", "aux.cu", "pool.cu", "sel_plan.cu", "tc.cu", "tc_bwd.cu", "tc_bwd_wide.cu", "tc_score.cu", "tc_fwdpair.cu", "tc_fwdpair_kernel.cu", "op.cu", "optim.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-DNSA_B200",
              "-Xptxas", "-v"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def _torch():
    import torch
    return torch


def _stamp():
    h = hashlib.sha256(_torch().__version__.encode())
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh", ".cpp")):
            h.update(open(os.path.join(CSRC, name), "rb").read())
    h.update(open(os.path.join(HERE, "..", "include", "nsa_b200.h"), "rb").read())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


EXT_OBJ = os.path.join(CSRC, "torch_op.o")


def _compile_ext():
    inc = os.path.join(os.path.dirname(_torch().__file__), "include")
    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include") if os.path.sep in _nvcc() else "/usr/local/cuda/include"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-D_GLIBCXX_USE_CXX11_ABI=%d" % _torch()._C._GLIBCXX_USE_CXX11_ABI,
           "-I" + inc, "-I" + os.path.join(inc, "torch", "csrc", "api", "include"), "-I" + sysconfig.get_paths()["include"],
           "-I" + cuda, '-DNSA_TORCH_VERSION="%s"' % _torch().__version__, "-c", os.path.join(CSRC, "torch_op.cpp"), "-o", EXT_OBJ]
    try:
        return subprocess.run(cmd, capture_output=True, text=True)
    except OSError as e:                       # no host compiler by that name
        return subprocess.CompletedProcess(cmd, 1, "", str(e))


def _link_ext(r):
    if r.returncode == 0:
        home = os.path.join(os.path.dirname(_torch().__file__), "lib")
        r = subprocess.run(["g++", "-shared", "-o", EXT, EXT_OBJ, "-L" + CSRC, "-l:libnsa_b200.so", "-Wl,-rpath,$ORIGIN",
                            "-L" + home, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-ltorch"],
                           capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        if os.path.exists(EXT):
            os.remove(EXT)
        print("warning: _nsa_torch.so could not be built: calls go through the Python nodes", file=sys.stderr)


def build_library(force=False, verbose=False):
    """Compile every .cu under csrc/ and link libnsa_b200.so; then _nsa_torch.so, which the package can do without: where
    it does not build, a warning says so.  Skips the work when the sources are unchanged since the last build.  Returns
    the library path."""
    stamp_file = os.path.join(CSRC, ".build_stamp")
    stamp = _stamp()
    if not force and os.path.exists(LIB) and os.path.exists(stamp_file) and open(stamp_file).read() == stamp:
        if not os.path.exists(EXT):
            _link_ext(_compile_ext())
        return LIB
    objs = [os.path.join(CSRC, src[:-3] + ".o") for src in SOURCES]

    def compile_one(src, obj):
        cmd = [_nvcc()] + NVCC_FLAGS + ["-c", os.path.join(CSRC, src), "-o", obj]
        return subprocess.run(cmd, capture_output=True, text=True)

    with ThreadPoolExecutor(max_workers=min(len(SOURCES) + 1, os.cpu_count() or 1)) as pool:
        ext = pool.submit(_compile_ext)
        results = list(pool.map(compile_one, SOURCES, objs))
    log = [r.stderr for r in results]
    for src, r in zip(SOURCES, results):
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("nvcc failed on " + src)
    r = subprocess.run([_nvcc(), "-shared", "-o", LIB] + objs + ["-lcudart"], capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("link failed")
    _link_ext(ext.result())
    with open(os.path.join(CSRC, "ptxas.log"), "w") as f:
        f.write("\n".join(log))
    with open(stamp_file, "w") as f:
        f.write(stamp)
    if verbose:
        print("\n".join(log))
    return LIB


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
