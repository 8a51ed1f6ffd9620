"""The D-step's transform of Y3 from its kept rows alone (k_y3fwd for the register lengths,
cuFFT rows of Lg / 4 for the others, bins 0 .. Lg/8 stored and mirrored by the solve)
against the FP64 oracle: every register length, kept-row counts that are odd, prime and
one, an odd and a single filter, more filters than the pipelined solve holds."""
import glob
import os
import re

import numpy as np
import pytest

from oracle import cdl_oracle as O

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-4            # the parity tolerance after a fixed iteration count
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cdlmotif.jl_gb300", "csrc")
LENGTHS = sorted({int(a) * int(p) for f in glob.glob(os.path.join(CSRC, "dstream_v*.cu"))
                  for a, p in re.findall(r"VARIANT\((\d+),\s*(\d+)", open(f).read())})
# (N, L, M, W): each register length with an odd M, then other lengths
SHAPES = [(3, lg // 4 - 4, 3, 2) for lg in LENGTHS] + \
    [(5, 112, 1, 6), (3, 15, 5, 2), (4, 13, 1, 3), (2, 61, 7, 5), (3, 99, 2, 1), (2, 30, 130, 3), (1, 1, 2, 1)]


@pytest.mark.parametrize("shape", SHAPES)
def test_dictionary_steps_against_oracle(pkg, built_lib, shape):
    N, L, M, W = shape
    Lg = 4 * L + 8 * W
    synth = pkg.synth
    S = synth.onehot(np.random.default_rng(L).integers(0, 4, size=(N, L)).astype(np.uint8))
    X0, D0 = synth.init_X0(9, N, M, Lg), synth.init_D0_unit_norm(9, M, Lg, 4 * W)
    setup = pkg.CDLSetup(M=M, filter_size=W, lambda_=0.1, rho=1.0, sigma=100.0)
    ref = O.init_cdl(S, M, W, 1.0, 100.0, 0.1, X0=X0, D0=D0)
    with pkg.init_cdl(setup, S, X0=X0, D0=D0) as c:
        pkg.code_update(c, 2)
        pkg.dict_update(c, 2)                    # the first from the initial spectra
        got = {f: c.get(f) for f in ("G1", "G3", "d", "g1", "g3", "Td", "G2")}
    O.code_update(ref, 2)
    O.dict_update(ref, 2)
    for f, v in got.items():
        want = getattr(ref, f)
        assert np.linalg.norm(v - want) <= TOL * max(np.linalg.norm(want), 1e-3), (f, rel(v, want))
