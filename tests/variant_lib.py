"""Builds of the library with another constant in one source, for paths that a run seldom or never takes."""
from __future__ import annotations

import ctypes
import os
import subprocess

from cudapathtracing_gb300 import build


def variant(tmp, sources: dict) -> ctypes.CDLL:
    """libcpt.so with `sources` ({file: [nvcc definitions]}) compiled anew; the other objects are the build's."""
    build.build()
    jobs, objs = [], []
    for src in build.SOURCES:
        stem = os.path.splitext(src)[0]
        if src not in sources:
            objs.append(os.path.join(build.OUT, stem + ".o"))
            continue
        objs.append(os.path.join(str(tmp), stem + ".o"))
        jobs.append(subprocess.Popen([build.NVCC, *build.ARCH, *build.COMMON, *sources[src], "-x", "cu", "-c",
                                      os.path.join(build.CSRC, src), "-o", objs[-1]]))
    assert all(j.wait() == 0 for j in jobs)
    lib = os.path.join(str(tmp), "libcpt_variant.so")
    subprocess.check_call([build.NVCC, *build.ARCH, "-shared", "-cudart", "static", "-o", lib, *objs])
    return ctypes.CDLL(lib)
