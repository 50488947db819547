"""Build recipe of libSOFIE_cuda.so (nvcc, sm_100a only) -- in-tree, no JIT cache.

The library is the product's only compute back end; nothing here falls back to a CPU path.
"""
from __future__ import annotations

import fcntl
import hashlib
import os
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = Path(__file__).resolve().parent / "csrc"
LIBDIR = Path(__file__).resolve().parent / "lib"
LIB = LIBDIR / "libSOFIE_cuda.so"
STAMP = LIBDIR / "libSOFIE_cuda.stamp"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-ffp-contract=off", "-I", str(ROOT / "include"), "-I", str(CSRC),
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: libSOFIE_cuda cannot be built")


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _fingerprint() -> str:
    h = hashlib.sha256()
    for p in sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + [ROOT / "include" / "sofie_cuda.h"]):
        h.update(p.name.encode())
        h.update(p.read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every .cu under csrc/ into one shared library. Re-uses an up-to-date build."""
    fp = _fingerprint()

    def current():
        return not force and LIB.exists() and STAMP.exists() and STAMP.read_text().strip() == fp
    if current():
        return LIB
    LIBDIR.mkdir(parents=True, exist_ok=True)
    # one builder at a time: the ranks of a multi-GPU job all arrive here; the first compiles, the rest wait
    with open(LIBDIR / ".build.lock", "a+") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if current():
                return LIB
            return _compile_and_link(fp, verbose)
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


def _compile_and_link(fp: str, verbose: bool) -> Path:
    objdir = LIBDIR / "obj"
    objdir.mkdir(exist_ok=True)
    nvcc = _nvcc()
    procs = []
    objs = []
    for src in sources():
        obj = objdir / (src.stem + ".o")
        objs.append(str(obj))
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}:\n{out}")
    tmp = LIB.with_name(f".{LIB.name}.{os.getpid()}.tmp")
    link = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", *objs, "-o", str(tmp), "-lcudart"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        tmp.unlink(missing_ok=True)
        raise RuntimeError(f"link of {LIB.name} failed:\n{r.stdout}")
    os.replace(tmp, LIB)
    STAMP.write_text(fp)
    return LIB


# ---- Python extension modules: the operator calls on torch tensors (over libSOFIE_cuda) and the calls of emitted Sessions ---------
CSRC_PY = Path(__file__).resolve().parent / "csrc_py"
OPS_LIB = LIBDIR / "_ops.so"
SESSION_LIB = LIBDIR / "_session.so"


def _build_extension(target: Path, sources: list[Path], tag: str, command) -> Path:
    """Run command(temporary output) unless `target` is the build of these sources and this tag."""
    import sysconfig
    h = hashlib.sha256(f"{tag} {sysconfig.get_config_var('EXT_SUFFIX')}".encode())
    for p in sources:
        h.update(p.read_bytes())
    fp, stamp = h.hexdigest(), target.with_suffix(".stamp")

    def current():
        return target.exists() and stamp.exists() and stamp.read_text().strip() == fp
    if current():
        return target
    LIBDIR.mkdir(parents=True, exist_ok=True)
    with open(LIBDIR / f".{target.stem}.lock", "a+") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if current():
                return target
            tmp = target.with_name(f".{target.name}.{os.getpid()}.tmp")
            r = subprocess.run(command(tmp), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
            if r.returncode != 0:
                tmp.unlink(missing_ok=True)
                raise RuntimeError(f"building {target.name} failed:\n{r.stdout}")
            os.replace(tmp, target)
            stamp.write_text(fp)
            return target
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


def build_ops() -> Path:
    """csrc_py/ops_native.cpp against the installed torch (headers and libraries) and libSOFIE_cuda."""
    import torch
    lib = build()
    src = CSRC_PY / "ops_native.cpp"

    def command(out):
        import sysconfig
        from torch.utils import cpp_extension
        cuda = Path(_nvcc()).resolve().parent.parent
        inc = [*cpp_extension.include_paths(), str(cuda / "include"), sysconfig.get_paths()["include"], str(ROOT / "include")]
        libs = cpp_extension.library_paths()
        return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                *[f for d in inc for f in ("-isystem", d)], str(src), "-o", str(out), *[f"-L{d}" for d in libs], f"-L{lib.parent}",
                "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-lSOFIE_cuda", "-Wl,-rpath,$ORIGIN",
                *[f"-Wl,-rpath,{d}" for d in libs]]
    return _build_extension(OPS_LIB, [src, ROOT / "include" / "sofie_cuda.h"], torch.__version__, command)


def build_session() -> Path:
    """csrc_py/session_native.c: Python's headers alone."""
    import sysconfig
    src = CSRC_PY / "session_native.c"
    return _build_extension(SESSION_LIB, [src], "", lambda out: ["gcc", "-O2", "-fPIC", "-shared", "-I", sysconfig.get_paths()["include"], str(src), "-o", str(out)])


_loaded = {}


def _load_extension(name: str, build_it):
    if name not in _loaded:
        import importlib.machinery
        import importlib.util
        path = str(build_it())
        spec = importlib.util.spec_from_file_location(name, path, loader=importlib.machinery.ExtensionFileLoader(name, path))
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        _loaded[name] = module
    return _loaded[name]


def load_ops():
    """The operator calls (built first when absent or stale); torch is imported before them, libSOFIE_cuda with them."""
    return _load_extension("_ops", build_ops)


def load_session():
    return _load_extension("_session", build_session)


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
