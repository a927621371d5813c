"""The LAZ decoder's warp keeps its models in shared memory, where one lane
stores what another loads for the next symbol. A missing barrier shows in no
test run as long as the lanes stay together, so the source is looked at: every
store of a symbol lies between two warp barriers, after the loads of this
symbol and before those of the next."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "potreeconverter_b200", "csrc")


def test_symbol_stores_lie_between_warp_barriers():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "laz_warp.cuh")).read())
    stores = list(re.finditer(r"m\.st_lane\([^;]*;\s*m\.st_lane\([^;]*;([^;]*;)", text))
    assert len(stores) == 2  # a model of up to 33 symbols, and one of more
    for group in stores:
        assert group.group(1).strip() == "__syncwarp();"
        function = text[text.rindex("__device__", 0, group.start()):group.start()]
        assert "__syncwarp();" in function[function.rindex("m.ld("):], function
    # symbols 31 and 32
    assert re.search(r"__syncwarp\(\);\s*if \(s > 30 && lane == 0\) b\.st\(", text)
