"""The order of the steps with which the upsampler's kernels let the next one in, in the source: a
mistake there could only show as a hang."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rosy_gb300", "csrc", "rz_upsample.cu")


def kernels():
    """Name and body of every kernel (bodies end at a brace in the first column), comments removed."""
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    return [(m.group(1), text[m.end():text.index("\n}", m.end())])
            for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\([^{;]*\)\s*\{", text)]


def test_tensor_memory_is_held_before_the_next_kernel_may_start():
    """A CTA of the next kernel that takes its tensor memory first waits for this kernel while it holds it; this
    kernel's CTA on that SM would then wait for tensor memory for ever. So a kernel allows the next one only after
    the allocation (in the warp that makes it, or past the barrier after it), and allocates once what it frees."""
    seen = []
    for name, body in kernels():
        if "tmem_alloc(" not in body:
            continue
        assert body.count("tmem_alloc(") == 1 and body.count("tmem_dealloc(") == 1, name
        if "pdl_allow_next()" not in body:
            continue
        seen.append(name)
        alloc, allow, barrier = body.index("tmem_alloc("), body.index("pdl_allow_next()"), body.index("__syncthreads()")
        assert body.count("pdl_allow_next()") == 1 and alloc < allow, name
        assert allow > barrier or re.search(r"if \(warp == 0\) \{\s*tmem_alloc\([^;]*;\s*pdl_allow_next\(\);\s*\}", body), name
        assert body.index("pdl_wait_previous()") > barrier > alloc, name
    assert sorted(seen) == ["k_conv", "k_wgrad"]
