"""The tuning constants that the build offers (--define) are read by the sources."""
import glob
import os
import re

from custingeralg_b200 import build


def test_every_offered_constant_has_an_effect():
    names = re.findall(r"TC_[A-Z0-9_]+", build.__doc__)
    assert names
    text = "".join(open(f).read() for f in glob.glob(os.path.join(build.CSRC, "*.cu")))
    for n in names:
        assert f"#ifndef {n}\n#define {n} " in text, n
        assert re.search(r"= [^;\n]*\b%s\b" % n, text), n
