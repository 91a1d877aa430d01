"""What kernels that run at the same time promise each other, read from their source: a race between them shows in no run."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "beatsaberrl_b200" / "csrc"


def _sources():
    return {p.name: p.read_text() for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cuh")}


def test_arrivals_at_the_other_cta_release_at_cluster_scope():
    """An mbarrier arrival without a scope releases within its own CTA only.  One that hands rows to a thread of another CTA has
    cluster scope, as a release or behind a release fence of that scope in the same statement."""
    seen = 0
    for name, text in _sources().items():
        for stmt in re.findall(r"asm volatile\((.*?);\s*\n(?:\}|  asm|  return)", text, re.S):
            for op in re.findall(r"mbarrier\.arrive[\w.:]*", stmt):
                if "shared::cluster" not in op:
                    continue
                seen += 1
                assert ".cluster.shared::cluster" in op, (name, op)
                assert ".release." in op or re.search(r"fence\.(release|acq_rel)[\w.:]*\.cluster", stmt), (name, op)
    assert seen >= 1


def test_barriers_of_both_ctas_are_awaited_at_cluster_scope():
    """Every barrier that mbar_arrive_cluster arrives at, or st.async counts on, is waited for with an acquire of cluster scope
    by the thread that goes on from it."""
    text = _sources()
    waits = {"gemm_res_tc5.cu": ["tmem_empty[buf]"], "gemm_pair_tc5.cu": ["tmem_empty[buf]"], "attn_block_tc5.cu": ["acc_empty[buf]"],
             "gemm_ln_tc5.cu": ["stats[buf]"], "block_tail_tc5.cu": ["x_ready", "h2_ready", "hid_ready["]}
    for name, src in text.items():
        if "mbar_arrive_cluster(map_to_cta" in src or "st_async_f2(map_to_cta" in src:
            assert name in waits, name
    for name, bars in waits.items():
        for bar in bars:
            calls = re.findall(r"(mbar_wait\w*|wait_epilogue|TAIL_WAIT\w*)(<[^>]*>)?\((?:smem_u32\()?&sh->" + re.escape(bar), text[name])
            assert calls, (name, bar)
            for fn, scope in calls:
                assert fn == "wait_epilogue" or scope in ("<true>", "<PAIR>", "<CL == 2>"), (name, bar, fn, scope)
    assert "return mbar_wait<PAIR>(bar, parity, abort);" in text["block_tail_tc5.cu"]
    assert "if (CLUSTER) wait_acquire_cluster();" in text["tc5.cuh"]
    assert re.search(r"wait_acquire_cluster\(\) \{ asm volatile\(\"fence\.acquire[\w.:]*\.cluster;", text["tc5.cuh"])


def test_copied_operands_go_to_a_kernel_that_waits_for_them():
    """Inside an overlapping sequence some kernels fetch their weight operand before their predecessor has ended, since weights
    are nobody's output.  The backward's transposed copies are: their products run on the warp-MMA kernel, which waits first."""
    struct = _sources()["train.cu"].split("struct Bwd {")[1].split("\n};")[0]
    for part in struct.split("transpose16(")[1:]:
        call = re.search(r"\b(linear\w*)\((?:a|r|f), st\)|transpose16\(", part)
        assert call is None or call.group(1) in (None, "linear_mma"), part[:200]
    body = _sources()["gemm_mma.cu"].split("linear_mma_kernel(LinearArgs p) {")[1]
    assert body.lstrip().startswith("pdl_begin();")


def test_a_cluster_loads_nothing_that_a_peer_may_already_be_writing():
    """The blocks' chain starts with loads into shared memory that peers send results into.  Step B's rows go to every CTA as soon
    as the heads' outputs are there, and with 2 H < 16 some CTA sends nothing before: nobody knows whether its loads have ended.
    So a warp loads only the columns of x that it sends itself (unit rank + 16 warp), after the cluster's only barrier."""
    kernel = _sources()["blocks_small.cu"].split("blocks_small_kernel(const __grid_constant__ Params args) {")[1]
    start = kernel.split("pdl_begin();")[1].split("cp_async_wait<0>();")[0]
    targets = re.findall(r"cp_async16\(base \+ l\.(\w+) \+ ([^,]*),", start)
    assert [t for t, _ in targets] == ["x", "h"], targets           # h is written by its own CTA only
    assert targets[0][1].startswith("u0 * UNIT32 + row32(row"), targets[0]
    assert re.search(r"if \(u0 < U\)\s*for \(int i = lane; i < 2 \* ROWS; i \+= 32\) \{[^}]*cp_async16\(base \+ l\.x", start)
    assert "const int u0 = rank + warp * CTAS" in kernel
    assert not re.search(r"(push_rows|send128)\w*\(base \+ l\.h\b", kernel)


def test_a_failed_count_of_resident_clusters_is_not_kept():
    """With no count the few-environment launches serve the call; one failed query must not decide that for the process."""
    body = _sources()["blocks_small.cu"].split("int chain::resident_clusters() {")[1].split("\n}")[0]
    failed = body.split("cudaGetLastError();")[1].split("}")[0]
    assert failed.strip().startswith("return 0;"), failed
    assert body.index("cudaGetLastError();") < body.index(".store(")


def test_residual_blocks_on_their_way_are_awaited_before_the_block_tail_exits():
    """A CTA that gives up a wait must not exit under copies into its shared memory: whatever a pre-store requested and did not
    consume -- a failed wait in the middle of it included -- is awaited, with a limit, buffer by buffer at the end."""
    src = _sources()["block_tail_tc5.cu"]
    prestore = src.split("auto prestore_tma = [&]")[1].split("    };\n")[0]
    assert "k = n_early; k < 3 && k < nb" in prestore and "if (k + 3 < nb) issue_block(t, k + 3);" in prestore    # three on their way
    failed = re.sub(r"\s+", " ", prestore.split("give_up(")[1].split("return false;")[0])
    assert "n_early = 3; for (int i = k; i < k + 3; ++i) if (i >= nb) io_phase ^= 1u << (i % 3);" in failed
    end = src.split("bounded, ignoring abort)\n    for (int k = 0; lane == 0 && k < n_early; ++k)")[1].split("bulk_wait_all();")[0]
    assert "io_full[warp - 2][k]), (io_phase >> k) & 1)" in end and "kSpinLimit" in end
