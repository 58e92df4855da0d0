"""Build librsfa_b200.so for sm_100a with nvcc, in-tree.

    python ascend-rsfa_b200/build.py [--force] [--verbose] [--trace]

Beside the library, the PyTorch side of the operator call (csrc/torch_binding.cpp) is
compiled against the installed torch into ascend_rsfa/_rsfa_torch*.so.  The library needs
no torch and is built without one; so does attention() run without the extension, 10 us
of host time slower.

The library lands beside the Python module that loads it
(ascend_rsfa/librsfa_b200.so) together with a stamp file holding a hash of the
sources, headers and compiler flags it was built from; a rebuild happens when
that hash no longer matches (file times are not consulted: the built library
travels with the source tree, and a checkout can carry any times), or with
--force.

--trace builds a separate debug library, ascend_rsfa/librsfa_b200_trace.so, with
-DRSFA_TRACE: the kernels of CTA 0 then log (clock, event code) pairs per role
into a buffer given through the "trace_ptr" option.  The per-role cycle tables
under profiles/ come from that build; the product library has no trace code.
"""
import hashlib
import importlib.util
import os
import re
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "ascend_rsfa", "librsfa_b200.so")
OUT_TRACE = os.path.join(HERE, "ascend_rsfa", "librsfa_b200_trace.so")
SOURCES = ["rsfa_api.cu", "fwd_generic.cu", "fwd_tcgen05.cu", "fwd_tcgen05_db.cu", "fwd_tcgen05_sp.cu", "fwd_short.cu"]
HEADERS = ["common.cuh", "ptx_sm100.cuh", "tcgen05_common.cuh", "tile_table.inc", os.path.join("..", "..", "include", "rsfa.h")]
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "-cudart", "static",
]


BINDING = "torch_binding.cpp"
OUT_BINDING = os.path.join(HERE, "ascend_rsfa", "_rsfa_torch" + sysconfig.get_config_var("EXT_SUFFIX"))
BINDING_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]
# what the extension is made from, beside the torch and the Python it is compiled against
BINDING_INPUTS = [os.path.join(CSRC, BINDING), os.path.join(HERE, "..", "include", "rsfa.h")]


def torch_home():
    """Directory of the installed torch, or None: no torch, or one without CUDA, which has no tensor to call with."""
    spec = importlib.util.find_spec("torch")
    if spec is None or spec.origin is None:
        return None
    home = os.path.dirname(spec.origin)
    return home if os.path.exists(os.path.join(home, "lib", "libc10_cuda.so")) else None


def torch_version(home):
    with open(os.path.join(home, "version.py")) as fh:
        return re.search(r"^__version__ = ['\"]([^'\"]+)['\"]", fh.read(), re.M).group(1)


def binding_command(home):
    """The g++ command line of the PyTorch extension: headers, libraries and C++ ABI of the torch in use."""
    import torch

    cuda = os.path.dirname(os.path.dirname(os.path.realpath(find_nvcc())))
    inc = [sysconfig.get_paths()["include"], os.path.join(home, "include"),
           os.path.join(home, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include")]
    return (["g++"] + BINDING_FLAGS +
            ["-D_GLIBCXX_USE_CXX11_ABI=%d" % torch.compiled_with_cxx11_abi(),
             '-DRSFA_TORCH_VERSION="%s"' % torch_version(home)] +
            ["-I" + i for i in inc] + [os.path.join(CSRC, BINDING), "-o", OUT_BINDING, "-L" + os.path.join(home, "lib")] +
            ["-l" + n for n in ("torch_python", "torch", "torch_cpu", "c10_cuda", "c10")])


def binding_hash(home):
    """Hash of the extension's sources and flags and of the torch and Python it is built against; no paths, so that a
    tree that moves to another machine with the same torch stays as it is."""
    h = hashlib.sha256()
    for f in BINDING_INPUTS + [os.path.join(home, "version.py")]:
        with open(f, "rb") as fh:
            h.update(fh.read() + b"\0")
    h.update(" ".join(BINDING_FLAGS).encode() + sys.version.encode())
    return h.hexdigest()


def build_binding(force=False):
    """The extension, or None where there is nothing to build it with: attention() then takes the ctypes route."""
    home = torch_home()
    if home is None:
        sys.stderr.write("no torch with CUDA here: %s is not built\n" % os.path.basename(OUT_BINDING))
        return None
    stamp = OUT_BINDING + ".stamp"
    want = binding_hash(home)
    if not force and os.path.exists(OUT_BINDING) and os.path.exists(stamp):
        with open(stamp) as fh:
            if fh.read().strip() == want:
                return OUT_BINDING
    if shutil.which("g++") is None:
        sys.stderr.write("no g++ here: %s is not built\n" % os.path.basename(OUT_BINDING))
        return None
    r = subprocess.run(binding_command(home), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout)
        raise RuntimeError("g++ failed on " + BINDING)
    with open(stamp, "w") as fh:
        fh.write(want + "\n")
    return OUT_BINDING


def find_nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC)")


def source_hash(flags):
    """Hash of everything the library is made from: sources, headers, flags."""
    h = hashlib.sha256()
    for f in SOURCES + HEADERS:
        with open(os.path.join(CSRC, f), "rb") as fh:
            h.update(f.encode() + b"\0" + fh.read() + b"\0")
    h.update(" ".join(flags).encode())
    return h.hexdigest()


def stale(out, flags):
    stamp = out + ".stamp"
    if not (os.path.exists(out) and os.path.exists(stamp)):
        return True
    with open(stamp) as fh:
        return fh.read().strip() != source_hash(flags)


def build(force=False, verbose=False, trace=False):
    out = build_library(force, verbose, trace)
    if not trace:
        build_binding(force)
    return out


def build_library(force=False, verbose=False, trace=False):
    out = OUT_TRACE if trace else OUT
    flags = FLAGS + (["-DRSFA_TRACE"] if trace else [])
    if not force and not stale(out, flags):
        return out
    nvcc = find_nvcc()
    objs = []
    build_dir = os.path.join(HERE, "build", "trace" if trace else "product")
    os.makedirs(build_dir, exist_ok=True)
    procs = []
    for src in SOURCES:
        obj = os.path.join(build_dir, src.replace(".cu", ".o"))
        cmd = [nvcc] + flags + (["-Xptxas", "-v"] if verbose else []) + ["-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, pr in procs:
        log, _ = pr.communicate()
        if verbose or pr.returncode != 0:
            sys.stderr.write(log)
        if pr.returncode != 0:
            raise RuntimeError("nvcc failed on " + src)
    link = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static",
            "-Xcompiler", "-fPIC", "-o", out] + objs
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout)
        raise RuntimeError("link failed")
    with open(out + ".stamp", "w") as fh:
        fh.write(source_hash(flags) + "\n")
    return out


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv, trace="--trace" in sys.argv))
