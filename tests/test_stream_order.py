"""A context's kernels run on its own non-blocking stream, which nothing orders after the
legacy stream: what they read has to be copied there.  A plain cudaMemcpy or cudaMemset
(legacy stream) is therefore allowed in the self-test only."""
import glob
import os
import re

from conftest import ROOT


def test_no_legacy_stream_copies_in_context_code():
    files = [f for f in glob.glob(os.path.join(ROOT, "da-gtm_gb300", "csrc", "*.cu*"))
             if not os.path.basename(f).startswith("selftest")]
    assert len(files) > 10
    found = [(os.path.basename(f), m) for f in files
             for m in re.findall(r"\bcuda(?:Memcpy|Memset|Memcpy2D)\s*\(", open(f).read())]
    assert not found
