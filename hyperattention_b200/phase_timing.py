"""Per-role cycle counters of the warp-specialised backward (and, with --forward, forward) kernel (a developer diagnostic, not
part of the product path).

    python hyperattention_b200/csrc/build.py --timing          # builds libhyperattn_b200_timing.so (-DHA_PHASE_TIMING)
    python -m hyperattention_b200.phase_timing [--heads 32] [--seq-len 131072]

Runs one non-causal forward + backward of the headline shape with the instrumented library and prints, per role of
attn_tc_bwd_ws_kernel (thread 0 of each role, averaged over the CTAs), how its cycles divide between waiting on each
barrier and working.  The counters use clock64 between the phases of every loop iteration; they perturb the kernel a
little, so the absolute kernel time is taken from bench.py, not from here.
"""
import argparse
import ctypes as C
import os

import torch

from . import _lib

EW = ['loop, item set-up', 'wait S^T / dP^T ready', 'lse / delta scaling, wait dS buffer free', 'loads, math, stores', 'store wait, fences, arrivals']
ISSUE = ['loop, item set-up', 'wait operand tile', 'wait inputs / accumulator', 'issue', 'tile done']
LOAD = ['row numbers', 'wait slot free', 'issue copies']
ROLES = {0: ('elementwise group 0', EW), 1: ('elementwise group 1', EW),
         2: ('drain group of dV', ['loop, item set-up', 'row numbers', 'wait accumulator complete', 'out of TMEM, staged, stored']),
         3: ('K loader', LOAD), 4: ('S^T warp', ISSUE), 5: ('dV warp', ISSUE), 6: ('dQ warp', ISSUE), 7: ('Q / dO loader', LOAD)}

# attn_tc_bwd_kt_kernel (head dim 128)
KT_ISSUE = ['loop, item set-up', 'wait K / V tile', 'wait unit', 'wait stage, accumulator', 'issue']
KT_ROLES = {0: ('elementwise group 0', ['loop, item set-up', 'wait S^T / dP^T ready', 'wait dS buffer free', 'loads, math, stores', 'store wait, fences, arrival']),
            2: ('drain group', ['loop, item set-up, row numbers', 'wait dQ', 'dQ out of TMEM, added', 'wait dV / dK', 'dV / dK out of TMEM, staged, stored']),
            3: ('K / V loader', ['row numbers', 'wait slot free', 'issue copies']), 4: ('S^T warp', KT_ISSUE), 1: ('dP^T warp', KT_ISSUE), 5: ('dV warp', KT_ISSUE),
            6: ('dQ warp', KT_ISSUE), 7: ('Q loader', LOAD)}

# attn_tc_fwd_kernel
FWD_ROLES = {0: ('softmax group 0', ['loop, item set-up', 'wait S ready', 'scores out of TMEM, maximum', 'exponentials, P, sum',
                                     'rescale, P store wait, arrival']),
             1: ('S warp of group 0', ['loop, item set-up', 'wait K tile', 'wait score buffer free', 'issue', 'tile done']),
             6: ('P V warp of group 0', ['loop, item set-up', 'wait V tile', 'wait P ready', 'issue', 'tile done']),
             2: ('K loader', ['index loads', 'wait slot free', 'issue copies']), 3: ('V loader', ['index loads', 'wait slot free', 'issue copies']),
             4: ('Q loader', ['index loads', 'wait slot free', 'issue copies']),
             5: ('epilogue group', ['item set-up', 'wait O complete', 'O out of TMEM', 'merge, stores'])}


def report(b, roles):
    for r, (name, phases) in roles.items():
        bb = b[:, r]
        tot = bb[:, :8].sum(1).mean().item()
        print(f'{name}: {round(tot)} cycles per CTA')
        for i, ph in enumerate(phases):
            print(f'   {ph:46s} {bb[:, i].mean().item():11.0f} {100 * bb[:, i].mean().item() / max(tot, 1):5.1f}%')


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument('--heads', type=int, default=32)
    ap.add_argument('--seq-len', type=int, default=131072)
    ap.add_argument('--forward', action='store_true', help='the forward kernel (attn_tc_fwd_kernel) instead of the backward')
    ap.add_argument('--dim', type=int, default=64)
    ap.add_argument('--causal', action='store_true', help='(forward) the last launch of a causal call; exact attention when --seq-len <= 2048')
    a = ap.parse_args()
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'libhyperattn_b200_timing.so')
    assert os.path.exists(path), 'build the instrumented library first: python hyperattention_b200/csrc/build.py --timing'
    _lib.LIB_PATH = path
    lib = _lib.load()
    from .module import HyperAttention
    torch.manual_seed(0)
    q, k, v, do = [torch.randn(1, a.heads, a.seq_len, a.dim, device='cuda', dtype=torch.bfloat16) for _ in range(4)]
    mod = HyperAttention(input_dim=a.dim).to(device='cuda', dtype=torch.bfloat16)
    buf = torch.zeros(4096 * 16, dtype=torch.int64, device='cuda')
    n_cta = min(148, a.heads * a.seq_len // 256)
    if a.forward:
        with torch.no_grad():
            mod(q, k, v, causal=a.causal)
            torch.cuda.synchronize()
            setter = lib.ha_debug_set_timing_buffer_fwd
            setter.restype, setter.argtypes = C.c_int, [C.c_void_p]
            setter(C.c_void_p(buf.data_ptr()))
            mod(q, k, v, causal=a.causal)
            torch.cuda.synchronize()
        print(f'{a.heads * a.seq_len // 256 / n_cta:.1f} work items per CTA (non-causal call)')
        report(buf.view(4096, 16).cpu().float()[:n_cta * 8].view(n_cta, 8, 16), FWD_ROLES)
        return
    qg, kg, vg = [t.clone().requires_grad_() for t in (q, k, v)]
    for rep in range(2):
        o = mod(qg, kg, vg, causal=a.causal)
        if rep == 1:
            setter = lib.ha_debug_set_timing_buffer_bwd_kt if a.dim == 128 else lib.ha_debug_set_timing_buffer_bwd_ws
            setter.restype, setter.argtypes = C.c_int, [C.c_void_p]
            setter(C.c_void_p(buf.data_ptr()))
        o.backward(do)
        torch.cuda.synchronize()
    b = buf.view(4096, 16).cpu().float()[:n_cta * 8].view(n_cta, 8, 16)
    report(b, KT_ROLES if a.dim == 128 else ROLES)


if __name__ == '__main__':
    main()
