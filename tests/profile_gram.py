"""The FP64 product by exact slices that the ncu summary under profiles/ profiles (pytest
does not collect this file): the overlap of 196 x 196 complex rows of 44^3 points
(k_ex_exp, k_ex_slice, k_ex_gemm, k_ex_reduce), twice.  It needs a GPU and the built
library.

  python tests/profile_gram.py
"""
import os
import sys
import time

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def main():
    import torch
    import filterbse_gb300 as F
    from filterbse_gb300 import workload as W
    g = W.Grid(44, 44, 44, 0.5, 0.5, 0.5, -11.0, -11.0, -11.0, 20.0)
    ctx = F.Context(g, np.zeros(g.ngrid), nspin=1, is_complex=True, precision=F.FP64)
    gen = torch.Generator(device="cuda:0").manual_seed(1)
    a, b = (torch.randn((196, ctx.stlen), dtype=torch.float64, device="cuda:0", generator=gen) for _ in range(2))
    for _ in range(2):
        t = time.time()
        ctx.gram(a, b)
        print(f"overlap: {time.time() - t:.4f}s")


if __name__ == "__main__":
    main()
