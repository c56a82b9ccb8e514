"""Launches that csipm_solve also records into its iteration graph (csrc/api.cu,
build_ipm_graph) run nothing while they are recorded, and a capture that fails
half way goes on with plain launches: recording must leave the solve's host
state as it was, so these functions take the handle const."""
import os
import re

API = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "compressedsensingipm.jl_b200", "csrc",
                   "api.cu")


def test_recorded_launches_take_a_const_handle():
    text = open(API).read()
    body = text[text.index("bool build_ipm_graph("):text.index("int ipm_graph_run(")]
    recorded = set(re.findall(r"\b(launch_(?!pdl)\w+)\(h,", body))
    assert recorded >= {"launch_resid_pass", "launch_corrector_start", "launch_step"}
    for name in recorded:
        decl = re.search(r"cudaError_t %s\(([^,]+)," % name, text)
        assert decl and decl.group(1).strip() == "const csipm_handle_s* h", name
    assert "rhs_due" not in body
