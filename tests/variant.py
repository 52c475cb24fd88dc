"""The library with some of its parts replaced, for tests that have to make a call
inside it fail: compiled sources that take the place of the library's objects of
the same name, or come beside them, and functions wrapped at link time."""
import os
import subprocess
import sys

from pike_gb300 import build as pk_build

HERE = os.path.dirname(os.path.abspath(__file__))


def link(out, sources, flags=(), wrap=()):
    """sources: paths; one named as a library source replaces that object."""
    objs = {s.rsplit(".", 1)[0]: os.path.join(pk_build.BUILD_DIR, s.rsplit(".", 1)[0] + ".o") for s in pk_build.SOURCES}
    if not all(os.path.exists(o) for o in objs.values()):
        pk_build.build(force=True)
    cc, where = pk_build.nvcc(), os.path.dirname(out)
    for s in sources:
        name = os.path.basename(s).rsplit(".", 1)[0]
        objs[name] = os.path.join(where, name + ".o")
        subprocess.run([cc, *pk_build.ARCH, *pk_build.NVFLAGS, *flags, "-c", s, "-o", objs[name]], check=True)
    subprocess.run([cc, *pk_build.ARCH, "-shared", "-o", out, *objs.values(),
                    *[x for w in wrap for x in ("-Xlinker", f"--wrap={w}")], "-lpthread"], check=True)
    return out


def run(child, *args):
    r = subprocess.run([sys.executable, os.path.join(HERE, child), *args], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.rstrip().endswith("ok"), r.stdout + r.stderr
