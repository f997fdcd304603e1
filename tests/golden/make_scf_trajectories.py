"""Writes scf_trajectories.json: the SCF trajectories of tests/test_scf_trajectories_gpu.py on a B200.

Run from the repository root as ``python tests/golden/make_scf_trajectories.py`` with the package whose
roundings are to be pinned.  The stored file comes from the kernels before the eigensolver of 2 to 16 bands, the
column density kernel and the constant-terms kernel were written for other callers.
"""

import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[2]))
sys.path.insert(0, str(Path(__file__).resolve().parents[1]))

import test_scf_trajectories_gpu as T  # noqa: E402

if __name__ == "__main__":
    out = {name: T.trajectory(name) for name in T.CASES}
    T.GOLD.write_text(json.dumps(out, indent=1) + "\n")
    print({k: v["iterations"] for k, v in out.items()})
