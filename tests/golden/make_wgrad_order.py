"""Writes wgrad_order.npz: elements of the convolutions' weight gradients, as the library in this
tree computes them on the GPU. The committed file comes from a build of commit 73410b6, whose
weight gradient ran on tcgen05.mma; run there with this file and ../test_gpu_wgrad_order.py."""
import importlib
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [os.getcwd(), os.path.dirname(HERE)]

if __name__ == "__main__":
    pkg = importlib.import_module("3dimagetoolkit_b200")
    import test_gpu_wgrad_order as T

    flat, x, t = T.step_inputs()
    with pkg.Context(0) as ctx, pkg.UNet(ctx, seed=1) as net:
        net.set_params(flat)
        g = T.samples(net.train_step(x, t, lr=0.0, want_grads=True)[1])
    np.savez_compressed(sys.argv[1] if len(sys.argv) > 1 else os.path.join(HERE, "wgrad_order.npz"), **g)
