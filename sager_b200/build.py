"""Builds sager_b200/libsager_b200.so from sager_b200/csrc/*.cu with nvcc for
sm_100a. The library is built in-tree (next to this file) so that it travels
with the source tree; nothing is installed. Every source file is compiled to
its own object (in parallel, only when it or a header changed) and the objects
are linked into the shared library. csrc/fastcall.c, the entry points as Python
callables, becomes an extension module of its own beside it."""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libsager_b200.so")
FASTCALL = os.path.join(HERE, "_fastcall" + sysconfig.get_config_var("EXT_SUFFIX"))      # (another interpreter does not load it)

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC,-fvisibility=hidden",
    "--expt-relaxed-constexpr", "--extended-lambda",
]
LINK_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-cudart", "static",
              "-Xcompiler", "-fPIC"]


def nvcc_path() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def sources():
    """CUDA sources and the host-only C++ sources (compiled by the same nvcc as host code)."""
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cpp")))


def headers():
    return glob.glob(os.path.join(CSRC, "*.cuh")) + [os.path.abspath(__file__)] + \
        glob.glob(os.path.join(os.path.dirname(HERE), "include", "*.h"))


def _obj(src):
    return os.path.join(OBJ, os.path.splitext(os.path.basename(src))[0] + ".o")


def needs_build() -> bool:
    return _older(LIB, sources() + headers())


def _older(path, than) -> bool:
    return not os.path.exists(path) or any(os.path.getmtime(p) > os.path.getmtime(path) for p in than)


def needs_fastcall() -> bool:
    """The module's functions come from the headers by way of capi.py and this file."""
    return _older(FASTCALL, headers() + [os.path.join(CSRC, "fastcall.c"), os.path.join(HERE, "capi.py")])


def fastcall_calls() -> str:
    """The C functions of csrc/fastcall.c: one per parameter list that an int-returning entry point with a trailing
    stream has in the headers (letters of capi.kinds_of)."""
    from . import capi
    kinds = sorted({k for k in map(capi.kinds_of, capi.prototypes().values()) if k})
    types = {"p": "void*", "i": "int", "q": "long long", "z": "size_t", "f": "float", "d": "double"}
    take = {"p": "as_pointer(a[{i}], &x{i})", "i": "as_integer(a[{i}], INT_MIN, INT_MAX, &n{i})",
            "q": "as_integer(a[{i}], LLONG_MIN, LLONG_MAX, &n{i})", "z": "as_integer(a[{i}], 0, LLONG_MAX, &n{i})",
            "f": "as_double(a[{i}], &n{i})", "d": "as_double(a[{i}], &n{i})"}
    out = []
    for ks in kinds:
        args = ks[:-1]
        out.append(f"static PyObject* call_{ks}(PyObject* self, PyObject* const* a, size_t nargsf, PyObject* kw) {{\n  Call* c = (Call*)self;\n"
                   "  void* s;\n  int rc;")
        for i, k in enumerate(args):
            out.append(f"  void* x{i};" if k == "p" else f"  {'double' if k in 'fd' else 'long long'} n{i};")
        out.append(f"  TAKE(kw == NULL && PyVectorcall_NARGS(nargsf) == {len(args)});")
        out += ["  TAKE(" + take[k].format(i=i) + ");" for i, k in enumerate(args)]
        out.append("  TAKE(as_stream(&s));\n  Py_BEGIN_ALLOW_THREADS")
        params = ", ".join(types[k] for k in ks)
        values = ", ".join([f"x{i}" if k == "p" else f"({types[k]})n{i}" for i, k in enumerate(args)] + ["s"])
        out.append(f"  rc = ((int (*)({params}))c->fn)({values});\n  Py_END_ALLOW_THREADS\n  return finish(c, rc);\n}}")
    out.append("static vectorcallfunc call_of(const char* kinds) {")
    out += [f'  if (strcmp(kinds, "{ks}") == 0) return call_{ks};' for ks in kinds]
    out.append("  return NULL;\n}\n")
    return "\n".join(out)


def build_fastcall() -> None:
    """Without a C compiler or Python's headers there is no module, and ops.py makes its calls through ctypes."""
    cc = os.environ.get("CC") or shutil.which("gcc") or shutil.which("cc")
    include = sysconfig.get_paths()["include"]
    if cc is None or not os.path.exists(os.path.join(include, "Python.h")):
        sys.stderr.write("sager_b200: no C compiler or no Python.h; calls from Python go through ctypes\n")
        return
    os.makedirs(OBJ, exist_ok=True)
    with open(os.path.join(OBJ, "fastcall_calls.inc"), "w") as f:
        f.write(fastcall_calls())
    cmd = [cc, "-O2", "-Wall", "-shared", "-fPIC", "-fvisibility=hidden", "-I", include, "-I", OBJ,
           "-o", FASTCALL + ".tmp", os.path.join(CSRC, "fastcall.c"), "-lpthread"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("building the extension module failed")
    os.replace(FASTCALL + ".tmp", FASTCALL)


def build(force: bool = False, verbose: bool = False, ptxas_info: bool = False) -> str:
    if force or needs_build():
        build_lib(force, verbose, ptxas_info)
    if force or needs_fastcall():
        build_fastcall()
    return LIB


def build_lib(force: bool, verbose: bool, ptxas_info: bool) -> None:
    os.makedirs(OBJ, exist_ok=True)
    nvcc = nvcc_path()
    hdr_t = max(os.path.getmtime(p) for p in headers())
    inc = ["-I", CSRC, "-I", os.path.join(os.path.dirname(HERE), "include")]

    def compile_one(src):
        obj = _obj(src)
        if not force and not ptxas_info and os.path.exists(obj) and \
                os.path.getmtime(obj) > max(hdr_t, os.path.getmtime(src)):
            return src, 0, ""
        flags = list(NVCC_FLAGS)
        if src.endswith(".cpp"):
            # host arithmetic that must reproduce the reference's bytes: hardware FMA for the fused
            # operations the source spells out, and no other contraction
            flags[flags.index("-fPIC,-fvisibility=hidden")] = "-fPIC,-fvisibility=hidden,-mfma,-ffp-contract=off"
        cmd = [nvcc] + flags + (["-Xptxas", "-v"] if ptxas_info else []) + inc + ["-c", "-o", obj, src]
        if verbose:
            print(" ".join(cmd))
        res = subprocess.run(cmd, capture_output=True, text=True)
        return src, res.returncode, res.stdout + res.stderr

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        results = list(ex.map(compile_one, sources()))
    failed = [r for r in results if r[1] != 0]
    if failed:
        for _, _, log in failed:
            sys.stderr.write(log)
        raise RuntimeError("nvcc failed: " + ", ".join(os.path.basename(r[0]) for r in failed))
    if ptxas_info or verbose:
        for _, _, log in results:
            sys.stderr.write(log)
    # objects of sources that no longer exist must not be linked
    objs = [_obj(s) for s in sources()]
    for stale in set(glob.glob(os.path.join(OBJ, "*.o"))) - set(objs):
        os.remove(stale)
    res = subprocess.run([nvcc] + LINK_FLAGS + ["-o", LIB + ".tmp"] + objs, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("link failed")
    os.replace(LIB + ".tmp", LIB)          # a reader never sees a half-written library


if __name__ == "__main__":
    build(force="--incremental" not in sys.argv, verbose=True, ptxas_info="--ptxas" in sys.argv)
    print(LIB)
