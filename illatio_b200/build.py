"""Builds libillatio_b200.so in-tree with nvcc for sm_100a, and the native host operators (_hostops.so) over it with g++.

    python -m illatio_b200.build [--force] [--verbose]
"""
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libillatio_b200.so")
HOSTOPS = os.path.join(HERE, "_hostops.so")
SOURCES = ["lib.cu", "quant.cu", "mv.cu", "moe.cu", "mm_id.cu", "mvf.cu", "decode.cu", "mvt.cu", "mve.cu", "mmd.cu", "mm_q8.cu", "mm_q8_i8.cu", "chain.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden", "--expt-relaxed-constexpr",
]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def stale():
    if not os.path.exists(LIB) or not os.path.exists(HOSTOPS):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(HOSTOPS))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(HERE, "..", "include", "illatio_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    """Compile every .cu under csrc/ into one shared library; returns its path."""
    if not force and not stale():
        return LIB
    objs = []
    procs = []
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    for src in sources():
        obj = os.path.join(HERE, "build", os.path.basename(src)[:-3] + ".o")
        cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(out)
        if p.returncode:
            raise RuntimeError("nvcc failed on %s" % src)
    cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
    subprocess.check_call(cmd)
    build_hostops()
    return LIB


def build_hostops():
    """The CPython extension module over the library: torch's headers for tensors and streams, the library beside it."""
    import torch
    t = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [os.path.join(t, "include"), sysconfig.get_paths()["include"], os.path.join(cuda if os.path.isdir(cuda) else "/usr/local/cuda", "include")]
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"] + ["-I" + i for i in inc]
                          + [os.path.join(CSRC, "hostops.cpp"), "-o", HOSTOPS, "-L" + HERE, "-lillatio_b200", "-L" + os.path.join(t, "lib"),
                             "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"])


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
