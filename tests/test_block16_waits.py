"""The block product's give-up path, by its source: elect.sync, tcgen05.ld and the
MMAs' commits need a whole warp, so no lane may act on its own answer to a wait.
(The path needs a barrier that never completes, which is not something to run.)"""

import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "asc_cpp_b200",
                      "csrc", "spmm_block16_tc.cu")


def test_waits_answer_for_the_whole_warp():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    assert text.count("try_wait") == 1  # every wait is wait_bar
    body = text[text.index("bool wait_bar("):]
    body = body[:body.index("\n}\n")]
    assert "try_wait" in body
    returns = re.findall(r"return ([^;]*);", body)
    assert returns and all(r.startswith("__all_sync(0xffffffffu,") for r in returns), returns


def test_giving_up_waits_for_the_copies_in_flight():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    producers = text[text.index("if (warp < kProducerWarps) {"):text.index("uint32_t it = 0, itm = 0;\n    for")]
    # the last wait of the role: its own stage's copy, without the abort flag
    waits = re.findall(r"wait_bar\(([^;{]*)\)", producers)
    assert re.match(r"&s\.full\[p\], \(uses - 1\) & 1u, nullptr", waits[-1]), waits
