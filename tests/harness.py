"""Device test programs linked with the engine's objects: they call the
launchers that the C ABI does not export."""
import ctypes
import glob
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def link(tmp_path, name, source, without=()):
    """Compiles a .cu source against lpma_gb300/csrc, links it with the
    objects of the built library (but those named in without) and loads it."""
    from lpma_gb300 import build
    build.build()
    src, so = tmp_path / (name + ".cu"), tmp_path / (name + ".so")
    src.write_text(source)
    objs = [o for o in sorted(glob.glob(os.path.join(build.BUILD, "*.o"))) if os.path.basename(o) not in without]
    subprocess.check_call([build._nvcc()] + build.ARCH + build.FLAGS + ["-shared", "-o", str(so), str(src)] + objs)
    return ctypes.CDLL(str(so))
