"""The FP64 kernels of Kerr and Johannsen give the same bits on one lane per geodesic, two, and several
however the compiler contracts products and sums: compiled without contraction
(-fmad=false), where every kernel that left it to the compiler would round otherwise, they
still agree, and foort_gpu_positions retraces a launch of one with another."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

SCRIPT = """
import sys
import numpy as np
import foort_gb300
foort_gb300.LIB_PATH = sys.argv[1]
from foort_gb300 import abi, workloads

for metric, params in ((abi.METRIC_KERR, (0.9,)), (abi.METRIC_JOHANNSEN, (0.7, 1.5, 0.0, 0.0, 0.0)),
                       (abi.METRIC_JOHANNSEN, (0.7, 1.5, 0.3, 0.2, 0.1))):
    for integrator, rlog, tolerance in ((abi.INTEGRATOR_RK4, 1, 0.001), (abi.INTEGRATOR_VERLET, 1, 1e-5),
                                        (abi.INTEGRATOR_VERLET, 0, 0.001), (abi.INTEGRATOR_RK4, 0, 0.001)):
        d = workloads.base_desc(abi.PREC_FP64)
        d.metric_id, d.integrator_id, d.rlog, d.verlet_tol = metric, integrator, rlog, tolerance
        d.epsilon, d.timeout_max_steps = 0.1, 300
        d.diag_flags = abi.DIAG_FOUR_COLOR_SCREEN | abi.DIAG_CLOSEST_RADIUS | abi.DIAG_GEODESIC_POSITION
        d.geopos_output_steps, d.geopos_freq = 9, abi.UpdateFreq(1, 1, 0)
        keep = abi.attach_images(d, [abi.make_image(params, r=1000.0, theta=1.1, half_width=9.0)])
        for side in (21, 130):
            px = abi.square_pixels(side)
            got = {}
            for lanes in (1, 2, 0):
                with foort_gb300.Engine(d) as e:
                    e.set_lanes(lanes)
                    first = e.integrate(px)
                    got[lanes] = (first,) + e.positions(px, first)
            for lanes in (2, 0):
                for a, b in zip(got[lanes], got[1]):
                    assert a.tobytes() == b.tobytes(), (metric, params, integrator, rlog, side, lanes)
print("same")
"""


@pytest.mark.gpu
def test_fp64_kernels_agree_without_contraction(tmp_path):
    from foort_gb300 import build
    build.build()
    apart = ("k_fp64_kerr.cu", "k_fp64_joh.cu", "k_split_kerr.cu", "k_split_joh.cu")
    objects, compiles = [], []
    for name in sorted(os.listdir(build.BUILD)):
        source = name[:-2]
        if source in apart:
            objects.append(str(tmp_path / name))
            compiles.append(subprocess.Popen([build.nvcc()] + build.NVFLAGS + ["-fmad=false", "-c", os.path.join(
                build.CSRC, source), "-o", objects[-1]]))
        elif name.endswith(".o"):
            objects.append(os.path.join(build.BUILD, name))
    assert [p.wait() for p in compiles] == [0] * len(apart)
    lib = str(tmp_path / "libfoort_apart.so")
    subprocess.run([build.nvcc()] + build.ARCH + ["-shared", "-o", lib] + objects + ["-lcudart"], check=True)
    run = subprocess.run([sys.executable, "-c", SCRIPT, lib], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert run.stdout.strip().endswith("same"), run.stdout + run.stderr
