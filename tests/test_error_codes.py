"""A CUDA error keeps its own code and text on the way to the caller: no entry
translates cudaErrorInvalidValue, which a refused launch or attribute gives as
well, into an argument error of the scheme.  Checked in the sources, as no
argument that passes validation makes such a launch fail."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "finess_b200", "csrc")


def test_cuda_errors_are_not_translated():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h", ".cpp")):
            with open(os.path.join(CSRC, f)) as h:
                assert not re.search(r"==\s*cudaError(?!NotReady|_t)\w+\s*\)\s*return\s+\w*err\(\s*FIN_ERR_ARG", h.read()), f
