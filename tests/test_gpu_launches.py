"""Launches that overlap their predecessor's tail keep the stream's order: an
iteration gives the results of the same one with every launch synchronised
(CUDA_LAUNCH_BLOCKING, read when CUDA starts, hence a process each)."""
import os
import subprocess
import sys

import numpy
import pytest

pytestmark = pytest.mark.gpu

RUN = """
import sys, numpy
from kelvin_gb300 import _lib, systems
from kelvin_gb300.cc_utils import DeviceSolver
from kelvin_gb300.quadrature import ft_quad
prec, digits, out = int(sys.argv[1]), int(sys.argv[2]), sys.argv[3]
ctx = _lib.context(0)
s = systems.ueg_recipe(14, 4.0, 19, 0.5)
beta = 1.0 / s.T
ti, g, G = ft_quad(6, beta, "lin")
sv = DeviceSolver.from_system(ctx, s.g_energies_tot(), s.g_fock_tot(), s.g_aint_tot(), beta, s.mu,
                              ti, g, G)
ctx.set_precision(prec, digits)
sv.spin_blocks(True)
sv.guess(1)
hist = [sv.step(0.5) for _ in range(8)]
T1, T2 = sv.amplitudes()
numpy.savez(out, T1=T1, T2=T2, E=numpy.array([h[0] for h in hist]))
"""


# Both runs make the same roundings but for the order of FP64 additions into
# one element (K cut over blocks); eight damped steps of a contracting
# iteration keep such differences near 1e-15 of the largest amplitude.
@pytest.mark.parametrize("prec,digits", [(0, 7), (1, 7), (1, 5)])
def test_overlapped_launches_match_synchronised_ones(tmp_path, prec, digits):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = []
    for blocking in ("0", "1"):
        out = str(tmp_path / ("r%s.npz" % blocking))
        env = dict(os.environ, CUDA_LAUNCH_BLOCKING=blocking, PYTHONPATH=root)
        subprocess.run([sys.executable, "-c", RUN, str(prec), str(digits), out], env=env, cwd=root,
                       check=True, timeout=120)
        res.append(numpy.load(out))
    a, b = res
    for k in ("T1", "T2", "E"):
        assert abs(a[k] - b[k]).max() <= 1e-12 * abs(b[k]).max()
