"""Argument types of the native library's entry points, so that calls pass plain Python numbers and addresses.

One letter per argument after the return type: p address (or stream), i int, u unsigned, l long, q long long, f float; s and v are
the return types text and nothing.  Without them every argument of every call is wrapped in a ctypes object of its own,
which took 3 of the 18 microseconds that the host needs for a small op.
"""
from __future__ import annotations

import ctypes

_TYPES = {"p": ctypes.c_void_p, "i": ctypes.c_int, "u": ctypes.c_uint, "l": ctypes.c_long, "q": ctypes.c_longlong,
          "f": ctypes.c_float, "s": ctypes.c_char_p, "v": None}

SIGNATURES = {
    "nsa_adamw8bit_multi": "ipipppiiifffffp",
    "nsa_adamw8bit_step": "ipppppppppliiifffffp",
    "nsa_adamw_multi": "ipipiiifffffp",
    "nsa_adamw_step": "ippppppliiifffffp",
    "nsa_affine_dequant": "ippppliip",
    "nsa_affine_quant": "ippppliiip",
    "nsa_attn_bwd": "ippppppppppiiiiiifiiiipppip",
    "nsa_attn_bwd_split": "ippppppppppiiiiiifiiiipppipppiiipiiiip",
    "nsa_attn_bwd_walks": "iiiiiiiii",
    "nsa_attn_bwd_walks_d64": "iiiiiiiii",
    "nsa_attn_fwd": "ipppppiiiiiifiiiipppip",
    "nsa_attn_importance": "ippppiiiiiifiiip",
    "nsa_comm_allgather": "ippliipuqip",
    "nsa_comm_reduce_scatter": "ippliifippuqp",
    "nsa_comm_reduce_scatter_parts": "i",
    "nsa_comm_rs_adamw8bit": "ippipppppppliififffffpuqp",
    "nsa_comm_signal": "ipiiup",
    "nsa_comm_wait": "ipiuqp",
    "nsa_conv1d_bwd": "ippppppppiiiiliip",
    "nsa_conv1d_bwd_parts": "liii",
    "nsa_conv1d_fwd": "ippppiiiliip",
    "nsa_copy2d": "iplplllp",
    "nsa_cross_entropy": "ipppplillip",
    "nsa_embedding_bwd": "ipppplip",
    "nsa_embedding_fwd": "ippplilp",
    "nsa_enable_peer_access": "ii",
    "nsa_gate_combine_bwd": "ippppppppppppplip",
    "nsa_gate_combine_bwd_ex": "ippppppliipppppppppplip",
    "nsa_gate_combine_fwd": "ippppppplip",
    "nsa_gate_combine_fwd_ex": "ippppppliiplip",
    "nsa_gates": "iplplpipipplip",
    "nsa_gdn_post": "ipppppppppppppppppiiiiifp",
    "nsa_gdn_prep": "ippppppppppiiiiifp",
    "nsa_gdn_seq_bwd": "ippppppppppiiiiifp",
    "nsa_gdn_seq_fwd": "ipppppppppiiiiifp",
    "nsa_gemm_bf16": "ipppiiiiiiiiiiip",
    "nsa_gemm_bf16_ag": "ippiiiiipplliipipuqip",
    "nsa_gemm_bf16_splitk": "ipppiiiiiiiiip",
    "nsa_gemm_pair_clusters": "i",
    "nsa_gemm_select": "vi",
    "nsa_inverse_blocks": "ippppppiiiiiip",
    "nsa_inverse_chunks": "iiii",
    "nsa_ipc_alloc": "ilpp",
    "nsa_ipc_close": "ip",
    "nsa_ipc_free": "ip",
    "nsa_ipc_open": "ipp",
    "nsa_l2norm_bwd": "ipppplip",
    "nsa_l2norm_fwd": "ippplifp",
    "nsa_last_error": "s",
    "nsa_launch_count": "q",
    "nsa_launch_count_reset": "v",
    "nsa_mamba3_scan": "ipppppppiiiip",
    "nsa_pool_bwd": "ippiiiiip",
    "nsa_pool_fwd": "ippiiiliip",
    "nsa_rmsnorm_add_fwd": "ipppppplifp",
    "nsa_rmsnorm_bwd": "ippppppppppliip",
    "nsa_rmsnorm_bwd_ldg": "ipplppppppppliip",
    "nsa_rmsnorm_bwd_noalloc": "ipppppppppliip",
    "nsa_rmsnorm_bwd_parts": "ili",
    "nsa_rmsnorm_bwd_res": "ippppppppplip",
    "nsa_rmsnorm_fwd": "ippppplifip",
    "nsa_rmsnorm_fwd_ldg": "ipplppplifip",
    "nsa_rope": "ippppliiiip",
    "nsa_scale_bf16": "ippplip",
    "nsa_select_blocks": "ippliiiip",
    "nsa_sm_count": "i",
    "nsa_ssd_chunk_grad": "iplplplppppppppppppiiiiip",
    "nsa_ssd_chunk_out": "iplplplpppppiiiiip",
    "nsa_ssd_chunk_state": "iiplplppppiiiiip",
    "nsa_ssd_finish": "ipppppppppppppiiip",
    "nsa_ssd_grad_slots": "iiii",
    "nsa_ssd_state_bwd": "ippppiiilp",
    "nsa_ssd_state_fwd": "ipppppiiilp",
    "nsa_ssd_states": "iiplplpppiiiiip",
    "nsa_ssd_states_form": "iiii",
    "nsa_ssd_states_in_one": "iiii",
    "nsa_status_read": "ipi",
    "nsa_sumsq": "iplippip",
    "nsa_sumsq_parts": "i",
    "nsa_swiglu_bwd": "ippppplilllp",
    "nsa_swiglu_fwd": "ippplillp",
    "nsa_union_blocks": "ippppiiiiiiip",
}


def declare(lib: ctypes.CDLL) -> None:
    """Sets the types of every entry point that the library has (a partial build may lack some)."""
    for name, sig in SIGNATURES.items():
        fn = getattr(lib, name, None)
        if fn is not None:
            fn.restype = _TYPES[sig[0]]
            fn.argtypes = [_TYPES[c] for c in sig[1:]]
