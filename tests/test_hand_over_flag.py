"""How the kernels read the hand-over word, from their source.

Blocks of a running kernel set the word (`Header::use_standard`) while others read it.  Threads
of one block that read it each for themselves could disagree, take different branches and meet
different block barriers; no run shows that reliably.  So a kernel that sets the word reads it
through `handed_over()`, which gives the whole block one answer.
"""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    'project_aether_b200', 'csrc')
WORD = 'use_standard'


def _functions(text):
    """Bodies of the kernels and device functions of a source file, by name."""
    text = re.sub(r'//[^\n]*', '', text)
    text = re.sub(r'__launch_bounds__\(.*\)', '', text)
    found = {}
    for match in re.finditer(r'__(?:global|device)__[^;{}]*?(\w+)\s*\([^;{}]*\)\s*\{', text):
        depth, at = 1, match.end()
        while depth:
            depth += {'{': 1, '}': -1}.get(text[at], 0)
            at += 1
        found[match.group(1)] = text[match.end():at]
    return found


def test_kernels_that_set_the_hand_over_word_read_it_once_per_block():
    writers = {}
    for name in sorted(os.listdir(CSRC)):
        for function, body in _functions(open(os.path.join(CSRC, name)).read()).items():
            writes = re.findall(r'hdr->%s = 1|atomicExch\(&hdr->%s, 1\)' % (WORD, WORD), body)
            if writes:
                writers[function] = body.count(WORD) - len(writes)
    assert {'small_sort_kernel', 'bucket_tail_kernel', 'bucket_finish_kernel',
            'bucket_finish_large_kernel'} <= set(writers)
    assert {f: reads for f, reads in writers.items() if reads} == {}


def test_the_word_is_read_by_one_thread_and_shared_behind_a_barrier():
    functions = _functions(open(os.path.join(CSRC, 'common.cuh')).read())
    body = functions['handed_over']
    assert '__syncthreads_or(threadIdx.x == 0' in body and WORD in body
