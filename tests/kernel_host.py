"""The search kernel's headers rewritten for a host compiler.

Only what is CUDA's is replaced: the runtime's include by a header of
`tests/kernel_host/` (which gives the intrinsics a meaning), the few functions
that are inline assembly by calls into its namespace `host`, and the block's
shared memory by what that namespace hands out."""
import os
import re
import shutil

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cuda_a_star_gb300", "csrc")
HERE = os.path.join(ROOT, "tests", "kernel_host")

# Functions that are one asm statement -> their body here.
BODIES = {
    "uint64_t globaltimer_ns()": "{ return host::globaltimer(); }",
    "void cas128(": "{ host::cas128(addr, c0, c1, n0, n1, o0, o1); }",
    "uint32_t ld_acquire_u32(": "{ return host::load(p); }",
    "unsigned long long ld_acquire_u64(": "{ return host::load(p); }",
    "uint32_t ld_relaxed_u32(": "{ return host::load(p); }",
    "unsigned long long ld_relaxed_u64(": "{ return host::load(p); }",
    "void st_relaxed_u64(": "{ host::store(p, v); }",
    "void red_relaxed_add_u32(": "{ host::add(p, v); }",
    "void fence_acq_rel_gpu()": "{ host::fence(); }",
    "void cluster_sync()": "{ host::cluster_barrier(); }",
    "uint4 ld_cluster(": "{ return host::load_cluster(p, rank); }",
}
TEXTS = {
    "extern __shared__ uint4 g_dyn_smem[];": "#define g_dyn_smem (host::block_dynamic())",
    "    __shared__ CtaShared s;\n    return s;": "    return host::block_shared<CtaShared>();",
    "    __shared__ typename D::Ctx c;\n    return c;": "    return host::block_context<typename D::Ctx>();",
    'asm volatile("prefetch.global.L2 [%0];" ::"l"(a));': "(void)a;",
    'asm volatile("fence.acq_rel.gpu;" ::: "memory");': "host::fence();",
}


def _body(src, name, new):
    i = src.index("{", src.index(name))
    depth, k = 0, i
    while True:
        depth += (src[k] == "{") - (src[k] == "}")
        if depth == 0:
            return src[:i] + new + src[k + 1:]
        k += 1


def rewrite(dst, shim, edit=lambda name, text: text):
    """Writes the headers to directory `dst`, over the warp operations of
    kernel_host/`shim`; `edit(name, text)` may change a header first."""
    for name in ("device_common.cuh", "search.cuh", "plugin.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            s = edit(name, f.read())
        s = s.replace("#include <cuda_runtime.h>", '#include "%s"' % shim)
        for k, v in BODIES.items():
            if k in s and re.search(re.escape(k) + r"[^;]*?\{", s):
                s = _body(s, k, v)
        for k, v in TEXTS.items():
            s = s.replace(k, v)
        assert "asm" not in re.sub(r"//.*", "", s), name
        with open(os.path.join(dst, name), "w") as f:
            f.write(s)
    with open(os.path.join(CSRC, "engine_types.h")) as f:
        s = edit("engine_types.h", f.read())
    with open(os.path.join(dst, "engine_types.h"), "w") as f:
        f.write(s)
    for name in os.listdir(HERE):
        shutil.copy(os.path.join(HERE, name), dst)
