"""Plans are sized by the number of SMs the device reports, which a partitioned
GPU has fewer of; the GB300's 152 stands only for a query that fails."""
import os
import re

from gbhsolve import build


def test_no_plan_holds_the_number_of_sms():
    found = []
    for name in sorted(os.listdir(build.CSRC)):
        text = open(os.path.join(build.CSRC, name)).read()
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
        found += ["%s: %s" % (name, line.strip()) for line in text.split("\n") if re.search(r"\b152\b", line)]
    assert found == ["gbh_engine.cu: int nsm = 152;"], found
    text = open(os.path.join(build.CSRC, "gbh_engine.cu")).read()
    assert text.count("cudaDevAttrMultiProcessorCount") == 1
