"""Builds the CUDA library on demand. `make` builds libllark_b200.so (everything); `make serve` builds
libllark_serve.so: the GEMM core, the decode linears and the generation-path ops of the layer-list decoders, which is
all a native checkpoint needs. `ensure_built()` is what the command-line tools call first: it does nothing when a
library is there, otherwise it compiles the serve subset (a lock file keeps two first calls from racing); the native
functions in front of the library (csrc/calls.cpp) for the running interpreter likewise."""
import fcntl
import os
import subprocess
import sys
import sysconfig

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "llark_b200")
FULL = os.path.join(PKG, "libllark_b200.so")
SERVE = os.path.join(PKG, "libllark_serve.so")


def _sources_newer_than(lib, names):
    t = os.path.getmtime(lib)
    paths = [os.path.join(PKG, "csrc", n) for n in names] + [os.path.join(ROOT, "include", "llark_b200.h")]
    return any(os.path.exists(p) and os.path.getmtime(p) > t for p in paths)


# what the Makefile's SERVE_OBJ is compiled from, headers included
SERVE_SOURCES = ("gemm_tcgen05.cu", "gemv.cu", "skinny.cu", "attn_step.cu", "seq_ops.cu", "seq_mixers.cu", "seq_swa_mma.cu",
                 "seq_swa_tc.cu", "seq_delta.cu", "seq_latent.cu", "seq_moe.cu", "seq_decay.cu", "seq_chunk.cu", "common.cuh",
                 "skinny.cuh", "attn_step.cuh")


def calls_path():
    """Where the native functions of this interpreter are."""
    return os.path.join(PKG, "_calls" + sysconfig.get_config_var("EXT_SUFFIX"))


def _make(target):
    env = dict(os.environ)
    env["PATH"] = "/usr/local/cuda/bin:" + env.get("PATH", "")
    return subprocess.run(["make", "-j8", "-C", ROOT, f"PYTHON={sys.executable}", target], env=env, capture_output=True, text=True)


class _Lock:
    def __enter__(self):
        os.makedirs(os.path.join(ROOT, "build"), exist_ok=True)
        self.f = open(os.path.join(ROOT, "build", ".serve.lock"), "w")
        fcntl.flock(self.f, fcntl.LOCK_EX)

    def __exit__(self, *exc):
        self.f.close()


def _python_h():
    return os.path.join(sysconfig.get_paths()["include"], "Python.h")


def _calls_stale():
    so = calls_path()
    return os.path.exists(_python_h()) and (not os.path.exists(so) or _sources_newer_than(so, ("calls.cpp",)))


def _ensure_calls():
    """The native functions beside a library that is there; without them the package goes on through ctypes, and says so here."""
    if not _calls_stale():
        return
    try:
        with _Lock():
            r = _make(os.path.relpath(calls_path(), ROOT)) if _calls_stale() else None
        why = r.stderr[-1000:] if r is not None and r.returncode else ""
    except OSError as e:  # no make, a tree that cannot be written
        why = str(e)
    if why:
        sys.stderr.write(f"llark_b200: {os.path.basename(calls_path())} was not built, calls go through ctypes: {why}\n")


def ensure_built(verbose=False):
    """Path of a usable library; compiles the serve subset if there is none (or its sources are newer)."""
    if os.environ.get("LLARK_LIB_PATH"):
        return os.environ["LLARK_LIB_PATH"]
    for lib in (FULL, SERVE):
        if os.path.exists(lib) and not _sources_newer_than(lib, SERVE_SOURCES):
            _ensure_calls()
            return lib
    with _Lock():
        if os.path.exists(SERVE) and not _sources_newer_than(SERVE, SERVE_SOURCES):
            return SERVE
        r = _make("serve")
        if verbose or r.returncode != 0:
            sys.stderr.write(r.stdout[-4000:] + r.stderr[-4000:])
        if r.returncode != 0:
            raise RuntimeError("building libllark_serve.so failed")
    return SERVE


if __name__ == "__main__":
    print(ensure_built(verbose=True))
