"""Builds libx17ai_b200.so in-tree with nvcc for sm_100a, and the native launch path _hostcall (a CPython extension) with
the host compiler (no JIT cache: the built libraries travel with the source tree)."""
import os
import subprocess
import sys
import sysconfig
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
LIB = HERE / "libx17ai_b200.so"
# the suffix names the Python it was built for: another one does not load it
HOSTCALL = HERE / ("_hostcall" + sysconfig.get_config_var("EXT_SUFFIX"))
SOURCES = [CSRC / "api.cu", CSRC / "shim.cpp"]
HEADERS = sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.hpp")) + [HERE.parent / "include" / "x17ai_b200.h"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-std=c++17", "-O3", "-lineinfo",
    "--ftz=true", "--fmad=true",
    "-Xcompiler", "-fPIC", "-shared",
    "-Xptxas", "-v",
]


def needs_build() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    return any(p.stat().st_mtime > t for p in SOURCES + HEADERS)


def build(force: bool = False, verbose: bool = False) -> Path:
    build_hostcall(force)
    if os.environ.get("X17AI_B200_LIB"):
        return Path(os.environ["X17AI_B200_LIB"])
    if not force and not needs_build():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc, *NVCC_FLAGS, "-o", str(LIB), *map(str, SOURCES), "-ldl"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    log = res.stdout + res.stderr
    (HERE / "build.log").write_text(" ".join(cmd) + "\n" + log)
    if res.returncode != 0:
        sys.stderr.write(log)
        raise RuntimeError("nvcc failed building libx17ai_b200.so")
    if verbose:
        print(log)
    return LIB


def build_hostcall(force: bool = False) -> Path:
    """The native launch path (csrc/hostcall.cpp), a CPython extension over torch's headers. It reads torch's C++ objects, so
    it belongs to one version of torch: the binary carries the version and is rebuilt under another one (_lib.hostcall
    does not use it there)."""
    import torch
    src = CSRC / "hostcall.cpp"
    deps = (src, HERE.parent / "include" / "x17ai_b200.h")
    built_for = f"torch {torch.__version__};"
    if (not force and HOSTCALL.exists() and all(d.stat().st_mtime <= HOSTCALL.stat().st_mtime for d in deps)
            and built_for.encode() in HOSTCALL.read_bytes()):
        return HOSTCALL
    t = Path(torch.__path__[0])
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DX17_BUILT_FOR="{built_for}"',
           f"-I{t}/include", f"-I{t}/include/torch/csrc/api/include", f"-I{sysconfig.get_paths()['include']}",
           str(src), "-o", str(HOSTCALL), f"-L{t}/lib", "-ltorch_python", "-ltorch_cpu", "-lc10"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError(f"g++ failed building {HOSTCALL.name}")
    return HOSTCALL


def build_kernel_objects():
    """The cubin + meta.json kernel objects used by the tests (prebuilt so they travel with the tree)."""
    from . import kernel_objects
    for dim in (512, 4096):
        kernel_objects.build_rms_norm(dim)


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
