"""Builds the torch extensions under quick-mlp_b200/lib/torch_ext/: qmlp_cu.so, the TorchScript custom classes
torch.classes.qmlp_cu.* (csrc/torch/qmlp_cu.cpp) over the header-only C++ class layer and libqmlp_b200.so, and
qmlp_calls.so, the native call path of the Python package (csrc/torch/calls.cpp), which resolves the library at run time.
Host C++ only (no kernels in them); nvcc is not involved and no GPU is needed to build."""
import os

HERE = os.path.dirname(os.path.abspath(__file__))
LIBDIR = os.path.join(HERE, "lib")
OUTDIR = os.path.join(LIBDIR, "torch_ext")
INCLUDE = os.path.abspath(os.path.join(HERE, "..", "include"))


def _build(name, source, ldflags, verbose):
    from torch.utils import cpp_extension
    src = os.path.join(HERE, "csrc", "torch", source)
    out = os.path.join(OUTDIR, name + ".so")
    deps = [src, os.path.join(INCLUDE, "qmlp_b200.h")] + [os.path.join(INCLUDE, "qmlp", f) for f in os.listdir(os.path.join(INCLUDE, "qmlp"))]
    if os.path.exists(out) and os.path.getmtime(out) >= max(os.path.getmtime(p) for p in deps):
        return out
    os.makedirs(OUTDIR, exist_ok=True)
    # The extensions must share the process's libstdc++.so with libqmlp_b200.so and with PyTorch. A compiler wrapper that
    # links the C++ runtime statically (one is first on PATH in some images) would put a second, uninitialised copy of
    # it into them, and every library loaded after them would bind its stream and locale symbols to that copy.
    if os.path.exists("/usr/bin/g++"):
        os.environ["CXX"] = "/usr/bin/g++"
    cpp_extension.load(name=name, sources=[src], extra_include_paths=[INCLUDE], extra_cflags=["-O2", "-std=c++17"],
                       extra_ldflags=ldflags + ["-lstdc++"], with_cuda=True, is_python_module=False,
                       build_directory=OUTDIR, verbose=verbose)
    for junk in ("build.ninja", ".ninja_deps", ".ninja_log", os.path.splitext(source)[0] + ".o"):
        p = os.path.join(OUTDIR, junk)
        if os.path.exists(p):
            os.remove(p)
    return out


def build_calls(verbose=False):
    """The native call path; importing the package needs it."""
    return _build("qmlp_calls", "calls.cpp", ["-ltorch_python"], verbose)


def build(verbose=False):
    build_calls(verbose)
    return _build("qmlp_cu", "qmlp_cu.cpp", ["-L" + LIBDIR, "-lqmlp_b200", "-Wl,-rpath," + LIBDIR], verbose)


if __name__ == "__main__":
    print(build(verbose=True))
