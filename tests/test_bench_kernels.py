"""The bench's device times are sums over every kernel of the measured calls:
its lists name all that the library times on those paths."""
import importlib.util
import os
import re

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "sdhash_gb300", "csrc")

COPIES = {"k_stage_gather"}  # host inputs to the device: in the end-to-end figures
PLAIN_COMMIT = {"k_stream_commit", "k_feat_links", "k_stream_chain", "k_stream_emit"}  # without an index
INDEX = {"k_stream_commit_round", "k_stream_index_pred", "k_pred_dirty", "k_index_first_init", "k_stream_index_first",
         "k_stream_index_mark", "k_stream_commit_index", "k_index_first", "k_index_mark"}
BLOCK = {"k_stream_ranks", "k_block_digest"}


def timed(*files):
    names = set()
    for f in files:
        with open(os.path.join(CSRC, f)) as s:
            names |= set(re.findall(r'TIMED_LAUNCH(?:_ON)?\(c, "(k_\w+)"', s.read()))
    return names


def test_kernel_lists_are_complete():
    spec = importlib.util.spec_from_file_location("bench_lists", os.path.join(REPO, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    names = timed("sdbf_api.cu", "index_search.cu") - COPIES
    assert {"k_stream_ranks", "k_stream_tiles", "k_block_digest", "k_index_query"} <= names
    assert set(bench.IB_KERNELS) == names - PLAIN_COMMIT - {"k_index_query"}
    assert set(bench.IX_KERNELS) == BLOCK | {"k_index_query"}
    assert set(bench.KERNELS) == names - INDEX - {"k_block_digest", "k_index_query"}
