"""Several threads, a context each, in a process whose first calls they make:
what is asked of CUDA once a device is asked by all of them at the same
time, and graph reductions take turns."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import threading
import numpy as np
import oracle
from cases import lower_star_volume, random_complex
from openph_gb300 import api, complexes as cx

mats = [cx.rips_cube(16, seed=1), cx.rips_cube(70, seed=2), cx.lower_star_image(60, 70, seed=3, sigma=2.0),
        cx.lower_star_image(180, 190, seed=4, sigma=3.0), random_complex(20, 0.5, 0.4, 5),
        cx.rips(cx.points_circle(165, 2), 1.2), lower_star_volume(7, seed=6), cx.rips_torus(100, 30_000, seed=7)]
want = [oracle.twist(bm)[:2] for bm in mats]
start = threading.Barrier(8)
wrong = []

def work(k):
    try:
        with api.Context(0) as c:
            start.wait()
            for i in range(3 * len(mats)):
                b = (i + k) % len(mats)
                for algo in ("pms", "twist", "ph_row_parallel") if i < len(mats) else ("pms",):
                    low, ess, _ = c.reduce(mats[b], algo)
                    if not np.array_equal(low, want[b][0]) or algo == "pms" and not np.array_equal(ess, want[b][1]):
                        wrong.append((k, b, algo))
    except Exception as e:
        wrong.append((k, repr(e)))

threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
for t in threads:
    t.start()
for t in threads:
    t.join()
print(wrong)
assert not wrong
"""


def test_first_calls_of_a_process_by_threads(cuda_lib):
    root = Path(__file__).resolve().parents[1]
    for _ in range(2):
        r = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, timeout=120, cwd=root,
                           env={**__import__("os").environ, "PYTHONPATH": f"{root}:{root / 'tests'}"})
        assert r.returncode == 0, r.stdout + r.stderr
