"""Kernels that may start before their predecessor has ended (they call griddepcontrol.wait) read what it writes with coherent
loads only: no __ldg, and __restrict__ on no input but the weights.  Read from the sources: the wrong load gives the right
values as long as the line is not in the cache, so a run shows nothing."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "p40-kernel_b200", "csrc")


def functions():
    """name -> (whether it is a kernel, parameters, body) of every device function."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"__launch_bounds__\(.*?\)\s(?=\w)", "", re.sub(r"//[^\n]*", "", open(path).read()))
        for m in re.finditer(r"^(?:static )?(?:__host__ )?__(global|device)__ ", text, re.M):
            head, _, rest = text[m.end():].partition("{")
            name = re.search(r"(\w+)\(", head)
            if ";" in head or not name:             # a variable
                continue
            depth, end = 1, 0
            while depth:
                depth += {"{": 1, "}": -1}.get(rest[end], 0)
                end += 1
            out[name[1]] = (m[1] == "global", head[name.end():], rest[:end])
    return out


def test_early_kernels_read_coherently():
    fns = functions()
    early = {n: f for n, f in fns.items() if f[0] and "pdl_wait_prior_grid" in f[2]}
    assert {"gemv_stream_kernel", "gemm_mma_kernel", "gemv_ring_kernel", "fwht_quant_kernel", "kv_attn_kernel", "attn_tc_kernel", "gdn_step_kernel",
            "tc16_split_kernel", "gemv_repack_kernel"} <= set(early)
    for name, (_, params, body) in early.items():
        assert set(re.findall(r"const \w+ \*\s*__restrict__ (\w+)", params)) <= {"W"}, name
        assert "__ldg(" not in body, name
        for called in set(re.findall(r"\b(\w+)(?:<[^;()]*>)?\(", body)) & set(fns):
            if not fns[called][0] and called != "attn_redo":      # (the CUDA-core attention reads what the launch in front of the planes wrote)
                assert "__ldg(" not in fns[called][2] and "ld.global.nc" not in fns[called][2].replace("ld.global.nc.u16", ""), (name, called)
                assert not re.findall(r"const \w+ \*\s*__restrict__", fns[called][1]), (name, called)


def test_kernels_wait_before_they_let_the_next_launch_in():
    """A launch that starts early waits for one predecessor, which has therefore to be behind its own wait before it lets anybody in.  The many-token mat-mul
    relies on it without a wait of its own for the weights: the split in front of it has waited for whoever wrote them."""
    inviting = {n: f[2] for n, f in functions().items() if "pdl_launch_dependents(" in f[2]}
    assert {"tc16_split_kernel", "quant_q8_1_kernel", "fwht_quant_kernel", "attn_planes_kernel", "gemv_few_kernel", "gemv_stream_kernel", "kv_append_kernel"} <= set(inviting)
    for name, body in inviting.items():
        assert 0 <= body.find("pdl_wait_prior_grid(") < body.find("pdl_launch_dependents("), name
