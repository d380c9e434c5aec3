"""Copies and clears that stages depend on are ordered before them.

A context's stream is a non-blocking one, which does not wait for the legacy
stream: a plain cudaMemcpy or cudaMemset of what a stage reads (descriptors,
first CTAs, ledger pieces) has no order with it, and a copy from pageable
memory may return before its data has arrived."""
import os
import re

import numpy as np
import pytest

import binary2d as b2
from helpers import make_case

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "app-binary2d_gb300", "csrc")


def test_copies_and_clears_name_a_stream():
    text = open(os.path.join(CSRC, "api.cu")).read()
    assert re.search(r"cudaStreamCreateWithFlags\(&ctx->stream, cudaStreamNonBlocking\)", text)
    plain = [line.strip() for line in text.splitlines() if re.search(r"\bcuda(Memcpy|Memset)\(", line)]
    assert not plain, plain


@pytest.mark.gpu
def test_batch_retiled_between_advances():
    """A batch whose first CTAs change before every advance, and whose stage
    capacity grows behind a queued one, gives the bits of one that is left alone."""
    cases = [b2.presets.iso_disk(nb, 64, seed=30 + nb) for nb in (2, 5, 3)]
    runs = [b2.Run(m, h, p) for m, h, p, _ in cases]
    cons = [make_case(*c)[0] for c in cases]
    folds = [1, 2, 1, 2, 1, 40]                       # (40 x RK2: more than the 64 stages that fit at first)
    tilings = [(1, 0), (64, 0), (2, 9), (64, 33), (8, 8), (16, 0)]
    out = []
    for retile in (False, True):
        with b2.Runtime(runs, precision="fp32_comp") as rt:
            for k, c in enumerate(cons):
                rt.upload(k, c)
            for fold, (th, rows) in zip(folds, tilings):
                if retile and fold < 40:
                    rt.set_tile(0, th)
                    rt.set_strip_rows(rows)
                rt.advance_async(fold)
            rt.synchronize()
            out.append([rt.download(k)[0] for k in range(3)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
