"""The warp that orders a space's bodies finds its space in 32-bit arithmetic for every grid up to 2^31 spaces."""
import os
import re

import numpy as np

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hoomd_rs_b200", "csrc",
                       "hmc_kernels.cu")


def test_space_of_a_warp():
    with open(KERNELS) as f:
        body = f.read().split("k_order_spaces(", 1)[1]
    index = re.search(r"const uint32_t c = ([^,;]+), lane", body).group(1)
    expression = index.replace("256u / 32u", "256u // 32u").replace("u", "").replace("threadIdx.x", "t").replace(
        "blockIdx.x", "b").replace("blockDim.x", "d")
    wrap = np.uint32
    with np.errstate(over="ignore"):
        for space in (0, 7, 8, 2 ** 27 - 1, 2 ** 27, 2 ** 27 + 9, 2 ** 31 - 1):
            block = space // 8
            for lane in (0, 31):
                names = {"b": wrap(block), "d": wrap(256), "t": wrap(space % 8 * 32 + lane)}
                assert int(wrap(eval(expression, {}, names))) == space
