"""Every copy and memset of a context goes to its own stream.  That stream does not wait
for the default stream, where the synchronous calls go: a memset, a copy within the
device and the last part of a copy from pageable memory are still to come when they
return, and a kernel of the context may be ahead of them."""
import os
import re

from wcns_b200.build import CSRC


def test_no_copy_or_memset_on_the_default_stream():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        assert not re.findall(r"\bcuda(?:Memcpy|Memset|MemcpyToSymbol|MemcpyFromSymbol|Memcpy2D|Memcpy3D)\s*\(", code), name
