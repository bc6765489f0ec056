"""The index's host side (hb_index.cu) on the CPU: compiled by g++ against a
CUDA runtime whose device memory is the host's, with a limit, and against
launchers that do nothing but what the host code looks at afterwards.  It shows
what the host asks of the device -- allocations, copies, launches and their
buffers -- where memory runs out, which no GPU has to be filled up for."""
import ctypes
import os
import re
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
CSRC = os.path.join(ROOT, "harmony_b200", "csrc")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
HERE = os.path.dirname(os.path.abspath(__file__))


def available() -> bool:
    return shutil.which("g++") is not None and os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h"))


def stubs() -> str:
    """Empty definitions of the launchers hb_internal.hpp declares, but for those
    fake_cuda.cpp defines."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "hb_internal.hpp")).read())
    defined = set(re.findall(r"^\w[\w:<>\* ]*[ \*](\w+)\(", open(os.path.join(HERE, "fake_cuda.cpp")).read(), re.M))
    out = []
    for ret, name, params in re.findall(r"^(void|int|size_t)\s+(\w+)\(([^;{]*)\);", text, re.M):
        if name in defined or name in ("index_device", "search_in_scratch", "set_last_error"):
            continue
        args = ", ".join(p.split("=")[0].strip() for p in re.sub(r"\s+", " ", params).split(","))
        out.append(f"{ret} {name}({args}) {{ {'return 1;' if ret != 'void' else ''} }}")
    return "\n".join(out)


def build(folder) -> ctypes.CDLL:
    so = os.path.join(str(folder), "libhost.so")
    with open(os.path.join(str(folder), "stubs.inc"), "w") as f:
        f.write(stubs())
    flags = ["g++", "-std=c++17", "-O1", "-w", "-fPIC", "-I" + CUDA_INCLUDE, "-I" + CSRC, "-I" + str(folder)]
    jobs = [subprocess.Popen(flags + ["-c", "-x", "c++", src, "-o", os.path.join(str(folder), obj)])
            for src, obj in ((os.path.join(CSRC, "hb_index.cu"), "index.o"),
                             (os.path.join(HERE, "fake_cuda.cpp"), "fake.o"))]
    for j in jobs:
        assert j.wait() == 0
    # (Its own runtime also where the process holds CUDA's.)
    subprocess.check_call(["g++", "-shared", "-Wl,--no-undefined", "-Wl,-Bsymbolic", "-o", so] +
                          [os.path.join(str(folder), o) for o in ("index.o", "fake.o")])
    return ctypes.CDLL(so)
