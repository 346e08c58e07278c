"""The cache's page-locked status word, which the host clears at the start of a call, goes only to kernels
that the same call waits for: a kernel still in flight from an earlier frame could raise it in between, and a
call whose own kernels are fine would report that frame's timeout.  (A wait that gives up cannot be had on
purpose, so the rule is read from the source.)"""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nbounce_gb300", "csrc", "nb_cache.cu")


def test_host_cleared_word_only_in_functions_that_wait():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    # top-level definitions: from a line that starts one to the closing brace in the first column
    bodies = re.findall(r"^(?:static )?(?:int|void|cudaError_t) (\w+)\([^;{]*\{\n(.*?)^\}", text, re.S | re.M)
    users = {name: body for name, body in bodies if "&c->report->status" in body}
    assert {"nb_cache_infer", "rows_op"} <= set(users)
    for name, body in users.items():
        cleared, given = body.find("c->report->status = 0"), body.find("&c->report->status")
        assert 0 <= cleared < given < body.find("cudaStreamSynchronize"), name
    assert text.count("&c->report->status") == sum(b.count("&c->report->status") for b in users.values())
