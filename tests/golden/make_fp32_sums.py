"""Writes fp32_sums.npz from the library of the tree that is first in the path (needs a GPU):

    PYTHONPATH=<tree> python tests/golden/make_fp32_sums.py <output>

The committed file comes from the tree of commit f2d3add, whose kernels held one node per thread."""
import os
import sys

import numpy as np

sys.path.append(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import test_gpu_fp32_sums as T  # noqa: E402

out = {"euler_%d_%d_%d" % c: T.euler_derivative(*c, 0).astype(np.float32) for c in T.EULER}
out.update({"cylinder_%d_%d_%d" % c: T.cylinder_residuals(*c) for c in T.CYLINDER})
np.savez_compressed(sys.argv[1], **out)
