"""The NF4 search by cells of 1/16 (csrc/quant_math.cuh) against the count of thresholds."""

import os
import re

import numpy as np

import offload_adam_b200


def _thresholds():
    path = os.path.join(os.path.dirname(offload_adam_b200.__file__), "csrc", "quant_math.cuh")
    text = open(path).read()
    block = text[text.index("#define OAB_NF4_THRESHOLD_BITS"):].split("\n\n")[0]
    bits = [int(b, 16) for b in re.findall(r"0x([0-9a-f]{8})u", block)]
    assert len(bits) == 15
    return np.array(bits, dtype=np.uint32).view(np.float32)


def _cell(x):  # round to nearest even of 16 x, exact in fp32 for |x| <= 1
    return np.rint(np.float64(x) * 16).astype(int) + 16


def test_every_cell_holds_at_most_one_threshold_and_gives_the_count():
    thr = _thresholds()
    at = _cell(thr)
    assert len(set(at)) == 15 and at.min() >= 0 and at.max() <= 32
    below = np.array([(at < c).sum() for c in range(33)])
    own = np.full(33, np.inf, dtype=np.float32)
    own[at] = thr
    near = np.concatenate([(np.arange(-8, 9) * np.spacing(t) + t).astype(np.float32) for t in thr])
    edges = (np.arange(-32, 33) / 32).astype(np.float32)
    edges = np.concatenate([edges, np.nextafter(edges, np.float32(2)), np.nextafter(edges, np.float32(-2))])
    x = np.concatenate([near, edges, np.linspace(-1, 1, 200001, dtype=np.float32)])
    x = np.clip(x, np.float32(-1), np.float32(1))
    c = _cell(x)
    assert np.array_equal(below[c] + (x >= own[c]), (thr[None] <= x[:, None]).sum(1))
