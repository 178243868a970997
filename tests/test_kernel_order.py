"""What can be told without a GPU about how kernels are chosen and ordered. What the kernels' sources must say about programmatic dependent launch: a wrong order of trigger, wait and loads is a race that a
run on a GPU hardly ever shows."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "strict_b200", "csrc")


def kernels():
    """{name: (file, parameter list, body)} of every __global__ function, comments taken out."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\(([^{;]*)\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            out[m.group(1)] = (os.path.basename(path), m.group(2), text[m.end():end])
    return out


KERNELS = kernels()


def test_kernels_are_found():
    assert len(KERNELS) > 60 and "quantize_rows_kernel" in KERNELS and "gemm_f32_tc_kernel" in KERNELS


@pytest.mark.parametrize("name", ["quantize_rows_kernel", "quantize_rows_int8_kernel", "quantize_rows_int8_wide_kernel"])
def test_row_splits_trigger_after_their_wait(name):
    """The product behind a split reads weights before its own wait: it may start only when what came before the split, which may
    have written them, is complete."""
    body = KERNELS[name][2]
    assert 0 <= body.index("pdl_wait()") < body.index("pdl_trigger()")


# Inputs that no kernel of a step's chain writes. Loads through a const __restrict__ pointer may be moved in front of the dependency wait.
CONSTANTS = {"w", "sw", "bias", "col_scale", "gain", "g", "b", "ln_gain", "ln_bias", "table", "wte", "wpe", "wkv"}


@pytest.mark.parametrize("name", [n for n in KERNELS if "pdl_wait()" in KERNELS[n][2]])
def test_chain_inputs_are_not_declared_invariant(name):
    declared = set(re.findall(r"const \w+\s*\*\s*__restrict__ (\w+)", KERNELS[name][1]))
    assert declared <= CONSTANTS
    loads = re.findall(r"__ldg\(\(const \w+\*\)\(?(\w+)", KERNELS[name][2])
    assert set(loads) <= {"wrow"}


@pytest.mark.parametrize("name", ["gemm_f32_tc_kernel", "gemm_pair_kernel", "gemm_tmem_kernel"])
def test_bounded_waits_follow_the_dependency_wait(name):
    """The lane that issues products waits for operands with a bound; a long predecessor must not use the bound up."""
    body = KERNELS[name][2]
    issue = body[body.index("constexpr uint32_t idesc"):]
    assert 0 <= issue.index("pdl_wait()") < issue.index("mbar_wait(")


# the option `prefetch` = 0: no weight is requested before the dependency wait. The first request of each product kernel:
@pytest.mark.parametrize("name,request_", [("gemm_f32_kernel", "__ldcs("), ("gemm_f32_tc_kernel", "load_w(0, i)"), ("gemm_rows_kernel", "= in ? __ldcs("),
                                           ("gemm_rows_kernel", "load_w(s0)"), ("gemm_tmem_kernel", "tma_load_2d_hint(")])
def test_weights_wait_where_the_option_says_so(name, request_):
    body = KERNELS[name][2]
    wait = re.search(r"if \(!(a\.)?prefetch\) pdl_wait\(\);", body)
    assert wait and wait.start() < body.index(request_)


# a layer norm in front of the product is refused beyond the rows and columns that the row kernel norms, not left out
@pytest.mark.parametrize("M,K", [(9, 768), (4700, 768), (8, 1028)])
def test_norm_in_front_is_not_dropped(M, K):
    import ctypes as C
    from strict_b200 import native

    class Args(C.Structure):
        _fields_ = [("M", C.c_int64), ("N", C.c_int64), ("K", C.c_int64), ("x", C.c_void_p), ("ldx", C.c_int64), ("w", C.c_void_p), ("ldw", C.c_int64),
                    ("bias", C.c_void_p), ("y", C.c_void_p), ("ldy", C.c_int64), ("mode", C.c_int), ("act_pos", C.c_float), ("act_neg", C.c_float),
                    ("col_scale", C.c_void_p), ("alpha", C.c_float), ("ln_gain", C.c_void_p), ("ln_bias", C.c_void_p), ("ln_eps", C.c_float)]

    here = C.create_string_buffer(4096)  # stands for a context and for data: a refused call reads neither
    p = C.addressof(here)
    f = native.lib()._Z10k_gemm_f32P14strictb200_ctxRK11GemmF32Args
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_void_p]
    a = Args(M=M, N=3072, K=K, x=p, ldx=K, w=p, ldw=K, y=p, ldy=3072, alpha=1, ln_gain=p, ln_bias=p, ln_eps=1e-5)
    assert f(p, C.addressof(a)) == native.ERR_INVALID_ARG


# M, N, K, E4M3 weights, finished product -> the kernel of few rows takes it: both sides of the lines that its rule draws, all measured
@pytest.mark.parametrize("M,N,K,f8,finished,takes", [
    (16, 9472, 64, False, True, True), (9, 9473, 64, False, True, False), (9, 9473, 768, False, True, True), (16, 18945, 768, False, False, False),
    (8, 18944, 64, False, True, True), (8, 18945, 64, False, True, False), (8, 32768, 256, False, True, False), (8, 18944, 3072, False, True, True),
    (16, 8192, 28672, False, True, True), (8, 4096, 4104, False, False, False), (17, 64, 64, False, True, False),
    (16, 9472, 512, True, False, True), (16, 9488, 512, True, False, False), (16, 6144, 1280, True, False, False), (8, 6144, 1280, True, False, True),
    (8, 16384, 512, True, True, True), (8, 16384, 256, True, True, False), (8, 9472, 64, True, True, True), (1, 32768, 128, True, True, False)])
def test_rule_of_the_few_row_kernel(M, N, K, f8, finished, takes):
    import ctypes as C
    from strict_b200 import native
    rule = native.lib()._Z18sb_gemm_rows_takeslllbb
    rule.restype, rule.argtypes = C.c_bool, [C.c_int64] * 3 + [C.c_bool] * 2
    assert rule(M, N, K, f8, finished) == takes


# the same of the products of a decode chain and of the stream over many channels
@pytest.mark.parametrize("name,request_", [("norm_rows_kernel", "__ldcs("), ("residual_rows_kernel", "__ldcs("), ("gemm_f32_stream_kernel", "request(n)")])
def test_chained_weights_wait_where_the_option_says_so(name, request_):
    body = KERNELS[name][2]
    wait = re.search(r"if \(!(a\.)?prefetch\) pdl_wait\(\);", body)
    assert wait and wait.start() < body.index(request_)


# both sides of the lines that the rules of the chain draw
@pytest.mark.parametrize("rule,M,N,K,takes", [
    ("norm", 1, 4096, 1024, True), ("norm", 16, 9472, 128, True), ("norm", 17, 4096, 1024, False), ("norm", 16, 9473, 128, False), ("norm", 8, 4096, 1152, False),
    ("norm", 8, 4096, 1000, False), ("residual", 16, 1024, 4096, True), ("residual", 1, 1184, 16, True), ("residual", 17, 1024, 2048, False),
    ("residual", 8, 1185, 2048, False), ("residual", 8, 1024, 4112, False), ("residual", 8, 1024, 2056, False)])
def test_rules_of_the_chain(rule, M, N, K, takes):
    import ctypes as C
    from strict_b200 import native
    f = getattr(native.lib(), {"norm": "_Z18sb_norm_rows_takeslll", "residual": "_Z22sb_residual_rows_takeslll"}[rule])
    f.restype, f.argtypes = C.c_bool, [C.c_int64] * 3
    assert f(M, N, K) == takes


# A length that is read before the dependency wait may change under the reader: one thread reads it, and the block takes it from there
@pytest.mark.parametrize("name", ["attn_decode_kernel", "latent_attn_decode_kernel"])
def test_early_length_is_one_reading_for_the_block(name):
    body = KERNELS[name][2]
    early = body[:body.index("pdl_wait()")]
    at = [m.start() for m in re.finditer(r"ld_volatile_i32\(", early)]
    assert len(at) == 1
    stored = re.search(r"if \(threadIdx\.x == \d+\) (\w+) = ld_volatile_i32\([^;]*;(.*?)__syncthreads\(\);(.*)", early, re.S)
    assert stored and not re.search(r"\b%s\b" % stored[1], stored[2]) and re.search(r"\b%s\b" % stored[1], stored[3])


# The latent decode kernel's softmax warps and the warp that issues its products, as far as their barriers go. A poll tells by one bit whether the phase it asks for
# has ended: with one barrier for the weights of all tiles two of them may end between two polls, which then never succeed.
def test_latent_decode_weights_are_seen_in_every_order():
    body = KERNELS["latent_attn_decode_kernel"][2]
    n = int((re.search(r"\bbar_p\[(\d)\]", body) or [0, 1])[1])
    if n == 2:
        assert "mbar_init(smem_u32(&bar_p[i]), 128)" in body and "ready(&bar_p[np & 1], pr)" in body and "smem_u32(&bar_p[t & 1])" in body and "pr ^= np++ & 1" in body
    tiles, todo, seen = 6, [(0, 0, 0, (0,) * n)], set()
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        t, ns, np_, ended = state  # softmax tile, products S and O issued (and, as fast as can be, complete), phases that have ended
        after = []
        if t < min(ns, tiles) and (t < 2 or np_ > t - 2):  # the weights of tile t take the half that the product of tile t - 2 has read
            after.append((t + 1, ns, np_, tuple(e + (i == t % n) for i, e in enumerate(ended))))
        if ns > np_ and ended[np_ % n] % 2 != np_ // n % 2:
            after.append((t, ns, np_ + 1, ended))
        elif ns < tiles and ns <= np_ + 1:
            after.append((t, ns + 1, np_, ended))
        assert after or np_ == tiles, f"nobody can go on: softmax at tile {t}, {ns} scores and {np_} outputs issued"
        todo += after


# Key tiles that were requested for another length are let in and requested again: the barrier they complete on is back in its first phase afterwards
def test_latent_decode_reloads_for_another_length():
    text = open(os.path.join(CSRC, "latent.cu")).read()
    let_in = text[text.index("int let_in("):]
    assert 0 <= let_in.index("mbar_wait(bar, 0)") < let_in.index("mbar_arrive(bar)") < let_in.index("return err")
    body = KERNELS["latent_attn_decode_kernel"][2]
    again = re.search(r"err = let_in\(smem_u32\(&k_full\[0\]\[0\]\), n_early, .*?n_early = 0;", body, re.S)
    assert again and body.index("pdl_wait()") < again.start() and again.end() < body.index("mbar_expect_tx_warp(smem_u32(&q_full)")
    issue = body[body.index("constexpr uint32_t idesc_s"):]
    assert issue.index("wait(&q_full, 0, 20)") < issue.index("ready(&k_full")


# The merge of the key chunks inside a cluster: where the bounded wait ran out nothing is written, and the block stays until no other can still store into it
def test_merge_that_gave_up_stays_until_the_others_have_left():
    body = KERNELS["attn_decode_kernel"][2]
    merge = body[body.index("mbarrier.try_wait"):]
    gave_up = re.search(r"if \(\w*\(?!__all_sync\(0xffffffffu, done\)[^{]*\{(.*?)return;", merge, re.S)
    assert gave_up and gave_up.end() < merge.index("*(uint2*)(out +")
    assert 0 <= gave_up[1].index("barrier.cluster.arrive") < gave_up[1].index("barrier.cluster.wait")


# The first arrival at a cluster's barrier is of the .aligned form, which a warp has to execute together: lane 0 has set up barriers alone just before
@pytest.mark.parametrize("path", ["attention.cu", "common.cuh"])
def test_first_cluster_arrival_follows_a_warp_barrier(path):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, path)).read())
    at = [m.start() for m in re.finditer(r'asm volatile\("barrier\.cluster\.arrive\.release\.aligned;"', text)]
    assert len(at) == 1 and re.search(r"__syncwarp\(\);\s*$", text[:at[0]])


# an expired wait is reported by the code nearest to its cause, not by that of whoever waited for the one that gave up
def test_latent_decode_reports_the_code_nearest_to_the_cause():
    body = KERNELS["latent_attn_decode_kernel"][2]
    assert "if (err && atomicMin(&err_s, err) > err) { *(volatile int*)a.status = err;" in body and body.count("a.status") == 1
    assert body.index("err_s = INT_MAX") < body.index("__syncthreads()")


# The scratch of the fp32 products on SM pairs: the smaller one goes when the larger one is there, and what could not be had is not asked for by every product
def test_scratch_of_fp32_products_survives_a_refusal():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "gemm_f32_pair.cu")).read())
    body = text[text.index("bool planes_scratch("):]
    body = body[:body.index("\n}")]
    assert body.index("planes_refused) return false") < body.index("cudaMalloc(") < body.index("ctx->planes_refused = bytes") < body.index("cudaStreamSynchronize(") < body.index("cudaFree(ctx->planes)")
    for path, call in (("api.cu", "int strictb200_free("), ("model.cu", "int strictb200_kv_destroy("), ("model.cu", "int strictb200_model_destroy(")):
        text = open(os.path.join(CSRC, path)).read()
        body = text[text.index(call):]
        assert "planes_refused = SIZE_MAX" in body[:body.index("\n}")]


# rules ask the context for its SMs; the few that are told no context share one constant, and what they choose is taken on a part with that many only
def test_rules_do_not_assume_a_number_of_sms():
    for path in glob.glob(os.path.join(CSRC, "*.c*")):
        code = re.sub(r"//[^\n]*", "", open(path).read()).replace("constexpr int SB_SMS = 148;", "")
        assert not re.search(r"\b148\b", code), path
    text = open(os.path.join(CSRC, "model.cu")).read()
    body = text[text.index("bool chained_step("):]
    assert "sm_count >= SB_SMS" in body[:body.index("\n}")]


# the structures that tests hand to internal functions are those of the library: names, order and types of the members
@pytest.mark.parametrize("name", ["GemmF32Args", "LatentShape"])
def test_structures_of_the_tests_match_the_library(name):
    import ctypes as C
    import test_gpu_chained_rows as t
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "common.cuh")).read())
    body = text[text.index("struct %s {" % name):]
    body = body[body.index("{") + 1:body.index("};")]
    types = {"int64_t": C.c_int64, "int": C.c_int, "float": C.c_float}
    members = []
    for line in body.split(";"):
        m = re.match(r"(?:const )?(\w+)([ *].*)", line.strip(), re.S)
        if not m or "(" in line:
            continue
        for part in m[2].split(","):
            members.append((re.search(r"\w+", part)[0], C.c_void_p if "*" in part else types[m[1]]))
    assert members == t.__dict__[name]._fields_


# every kernel behind this entry reads its operands 16 bytes at a time: others are refused on the host
@pytest.mark.parametrize("M,off_x,off_w", [(1, 4, 0), (4, 0, 8), (300, 12, 0), (3000, 0, 4)])
def test_fp32_operands_that_are_not_aligned_are_refused(M, off_x, off_w):
    import ctypes as C
    from strict_b200 import native
    here = C.create_string_buffer(4096 + 16)  # stands for a context and for data: a refused call reads neither
    p = (C.addressof(here) + 15) // 16 * 16
    import test_gpu_chained_rows as t
    f = native.lib()._Z10k_gemm_f32P14strictb200_ctxRK11GemmF32Args
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_void_p]
    a = t.GemmF32Args(M=M, N=3072, K=768, x=p + off_x, ldx=768, w=p + off_w, ldw=768, y=p, ldy=3072, alpha=1)
    assert f(p, C.addressof(a)) == native.ERR_INVALID_ARG


# the blocks of fp32 prompt attention are dealt out when the product in front of the cache append has left its SMs
def test_cache_append_of_prompts_triggers_after_its_wait():
    body = KERNELS["kv_append_f32_vec_kernel"][2]
    assert 0 <= body.index("pdl_wait()") < body.index("pdl_trigger()")
