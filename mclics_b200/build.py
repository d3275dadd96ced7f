"""Builds libmclics_b200.so in-tree with nvcc for sm_100a (B200).

    python -m mclics_b200.build [--force]

Objects go to mclics_b200/_build/, the library to mclics_b200/libmclics_b200.so, the command-line program to
mclics_b200/mclics_b200. kernels_ref8.cu (the reference-order replay kernel) is compiled with -fmad=false so that
its arithmetic rounds like the reference's x86-64 build.
"""
import argparse
import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libmclics_b200.so")
EXE = os.path.join(HERE, "mclics_b200")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC,-O3", "--expt-relaxed-constexpr",
          "-I" + os.path.join(HERE, "..", "include")] + ARCH
PER_FILE = {"kernels_ref8.cu": ["-fmad=false"]}
# Sources compiled once per set of macros: {file: {object suffix: flags}}.
VARIANTS = {"sweep_pass_kernels.cu": {
    "%s%s%s%s" % (pot, "_chiral" * chiral, "_flip" * flip, "_field" * field):
        ["-DPASS_POT=POT_" + pot.upper()] + ["-DPASS_%s=%s" % (k, str(bool(v)).lower())
                                             for k, v in (("CHIRAL", chiral), ("FLIP", flip), ("FIELD", field))]
    for pot, chiral, flip, field in (("ghrl", 1, 1, 1), ("ghrl", 1, 0, 1), ("ghrl", 1, 0, 0), ("ghrl", 0, 1, 1),
                                     ("ghrl", 0, 0, 1), ("ghrl", 0, 0, 0), ("pear", 0, 1, 1), ("pear", 0, 1, 0),
                                     ("ll", 0, 1, 1), ("ll", 0, 0, 1), ("ll", 0, 0, 0))}}
SOURCES = ["sweep_pass_kernels.cu", "sweep_pass.cu", "sweep_resident_ghrl.cu", "sweep_resident_ghrl_chiral.cu",
           "sweep_resident_pear.cu", "sweep_resident_ll.cu", "sweep_fused_ghrl.cu", "sweep_fused_pear.cu",
           "sweep_fused_ll.cu", "learned.cu", "kernels.cu", "kernels_ref8.cu", "sweep_fused.cu", "observe_static.cu",
           "extras.cu", "engine.cpp", "driver.cpp"]  # slowest first: they start compiling first


def nvcc():
    for p in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if p and os.path.exists(p):
            return p
    raise RuntimeError("nvcc not found")


def _deps_newer(obj, src):
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    heads = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    heads.append(os.path.join(HERE, "..", "include", "mclics_b200.h"))
    return any(os.path.getmtime(p) > t for p in [src] + heads)


def _units():
    """(source, flags, object) of everything that is compiled."""
    out = []
    for src in SOURCES:
        if os.path.exists(os.path.join(CSRC, src)):
            for suffix, flags in VARIANTS.get(src, {"": []}).items():
                obj = src + ("." + suffix if suffix else "") + ".o"
                out.append((src, PER_FILE.get(src, []) + flags, os.path.join(BUILD, obj)))
    return out


def _compile(unit, verbose):
    src, flags, obj = unit
    path = os.path.join(CSRC, src)
    if not _deps_newer(obj, path):
        return obj
    cmd = [nvcc()] + COMMON + flags + ["-c", path, "-o", obj]
    if src.endswith(".cpp"):
        cmd[1:1] = ["-x", "cu"]
    if verbose:
        print(" ".join(cmd))
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s%s" % (src, r.stdout, r.stderr))
    return obj


def build(force=False, verbose=False):
    os.makedirs(BUILD, exist_ok=True)
    units = _units()
    if force:
        for _, _, obj in units:
            if os.path.exists(obj):
                os.remove(obj)
    with cf.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(lambda u: _compile(u, verbose), units))
    if force or not os.path.exists(LIB) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        cmd = [nvcc()] + ARCH + ["-shared", "-cudart", "static", "-o", LIB] + objs
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n%s%s" % (r.stdout, r.stderr))
    main_src = os.path.join(CSRC, "main.cpp")
    if os.path.exists(main_src) and (force or not os.path.exists(EXE) or os.path.getmtime(LIB) > os.path.getmtime(EXE)
                                     or os.path.getmtime(main_src) > os.path.getmtime(EXE)):
        cmd = [nvcc(), "-O2", "-std=c++17", "-I" + os.path.join(HERE, "..", "include"), main_src, "-o", EXE,
               "-L" + HERE, "-lmclics_b200", "-Xlinker", "-rpath,$ORIGIN"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("CLI link failed:\n%s%s" % (r.stdout, r.stderr))
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("-v", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.v))
    sys.exit(0)
