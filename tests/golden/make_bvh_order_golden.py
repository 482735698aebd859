"""Regenerates golden/bvh_order.npz: the leaf order (face ids) of the SAH build
on the soups of tests/test_bvh_order_gpu.py, from the checkout it is run in.
Needs the GPU:

    python tests/golden/make_bvh_order_golden.py

The file was recorded from the builder that split every small node with a
warp's bins (one warp a node, no chip-wide list); the order has not changed
since, so a run must reproduce it byte for byte.
"""

import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [os.path.dirname(HERE), os.path.dirname(os.path.dirname(HERE))]

from test_bvh_order_gpu import GOLDEN, SIZES, leaf_order  # noqa: E402

if __name__ == "__main__":
    orders = {f"n{n}": leaf_order(n) for n in SIZES}
    if os.path.exists(GOLDEN):
        old = np.load(GOLDEN)
        print("changed:", [k for k, v in orders.items() if k not in old or not np.array_equal(old[k], v)])
    np.savez_compressed(GOLDEN, **orders)
