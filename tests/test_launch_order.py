"""Where kernels let the next one start (launch_dependents) among their waits.

A small kernel between two large ones -- the padded copy of a call -- that lets its dependents go before
it has waited itself starts the chain behind it as well: the copies and evaluations of the calls to
come, while an earlier evaluation still runs.  It waits first."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "opensubdiv_gb300", "csrc")


def test_the_padded_copy_waits_first():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "stencils_batch.cu")).read())
    body = text[text.index("k_pad_one(const PadJob"):]
    body = body[:body.index("\n}")]
    assert 0 < body.index("wait_for_primary();") < body.index("launch_dependents();")
    assert body.index("launch_dependents();") < body.index("pad_row(")
