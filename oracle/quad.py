"""The CPU oracle in extended precision (``long double``: 113 bits on aarch64,
64 on x86_64), for tests that measure how far complex128 results are from the
true values.

TEST INFRASTRUCTURE ONLY, as ``oracle.py``.  The source is ``qg_oracle.c``
itself with its scalar type widened: ``double`` becomes ``long double``,
``<tgmath.h>`` picks the matching functions (it has no ``cexp``), and pi gets its further digits.
Angles and weights are the caller's doubles, exactly.
"""
import ctypes
import os
import subprocess

import numpy as np

from .oracle import BUILD_DIR, ENT_CNOT, HERE, PLACE_BEFORE, _chk, _p

LIB_PATH = os.path.join(BUILD_DIR, "libqg_oracle_quad.so")
_PI = "3.14159265358979323846"
_HEAD = ("#include <complex.h>\n#include <math.h>\n#include <stdint.h>\n#include <stdlib.h>\n#include <string.h>\n"
         "#include <tgmath.h>\n#ifdef _OPENMP\n#include <omp.h>\n#endif\n#define double long double\n#define cexp cexpl\n")

# bits of a result's fraction
BITS = np.finfo(np.longdouble).nmant


def build(force=False):
    src = os.path.join(HERE, "qg_oracle.c")
    newest = max(os.path.getmtime(src), os.path.getmtime(os.path.abspath(__file__)))
    if not force and os.path.exists(LIB_PATH) and os.path.getmtime(LIB_PATH) >= newest:
        return LIB_PATH
    os.makedirs(BUILD_DIR, exist_ok=True)
    text = open(src).read()
    assert text.count(_PI) == 1
    tmp = LIB_PATH + ".tmp%d" % os.getpid()
    with open(tmp + ".c", "w") as f:
        f.write(_HEAD + text.replace(_PI, _PI + "264338327950288L"))
    subprocess.run(["gcc", "-O2", "-fopenmp", "-fPIC", "-shared", "-std=c11", "-o", tmp, tmp + ".c", "-lm"], check=True)
    os.remove(tmp + ".c")
    os.replace(tmp, LIB_PATH)
    return LIB_PATH


_lib = None


def lib():
    global _lib
    if _lib is None:
        build()
        _lib = ctypes.CDLL(LIB_PATH)
        P, I = ctypes.c_void_p, ctypes.c_int
        for name, args in {
            "qgo_mcclean_run": [I, I, P, P, I, I, I, P, P, P, P, P, P, P],
            "qgo_mcclean_grad": [I, I, P, P, I, I, I, P, P, P, P, P, P, P],
            "qgo_mcclean_grad_uncompute": [I, I, P, P, I, I, I, P, P, P, P, P, P, P],
            "qgo_qaoa_run": [I, I, P, P, I, P, P, P, P, P, P, P],
            "qgo_qaoa_grad": [I, I, P, P, I, P, P, P, P, P, P, P],
            "qgo_qaoa_grad_uncompute": [I, I, P, P, I, P, P, P, P, P, P, P],
        }.items():
            f = getattr(_lib, name)
            f.argtypes, f.restype = args, ctypes.c_int
    return _lib


def _ld(a, dtype=np.longdouble):
    return None if a is None else np.ascontiguousarray(a, dtype=dtype)


def mcclean(n, axes, angles, terms, entangler=ENT_CNOT, placement=PLACE_BEFORE, ini=None, grad=True, uncompute=False):
    """(E, gradient or final state) of a McClean circuit, in long double."""
    axes, angles, w = np.ascontiguousarray(axes, np.int32), _ld(angles), _ld(terms.w)
    ini, E = _ld(ini, np.clongdouble), np.zeros(1, np.longdouble)
    out = np.zeros(angles.shape, np.longdouble) if grad else np.zeros(2 ** n, np.clongdouble)
    f = lib().qgo_mcclean_run if not grad else lib().qgo_mcclean_grad_uncompute if uncompute else lib().qgo_mcclean_grad
    _chk(f(n, axes.shape[0], _p(axes), _p(angles), entangler, placement, len(terms), _p(terms.kind), _p(terms.q0),
           _p(terms.q1), _p(w), _p(ini), _p(E), _p(out)))
    return E[0], out


def qaoa(n, betas, gammas, terms, ini=None, grad=True, uncompute=False):
    """(E, gradient [p, 2] or final state) of a QAOA circuit, in long double."""
    betas, gammas, w = _ld(betas), _ld(gammas), _ld(terms.w)
    ini, E = _ld(ini, np.clongdouble), np.zeros(1, np.longdouble)
    out = np.zeros((len(betas), 2), np.longdouble) if grad else np.zeros(2 ** n, np.clongdouble)
    f = lib().qgo_qaoa_run if not grad else lib().qgo_qaoa_grad_uncompute if uncompute else lib().qgo_qaoa_grad
    _chk(f(n, len(betas), _p(betas), _p(gammas), len(terms), _p(terms.kind), _p(terms.q0), _p(terms.q1), _p(w),
           _p(ini), _p(E), _p(out)))
    return E[0], out
