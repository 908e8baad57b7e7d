// The shapes that decode kernels are built for, one FB_DECODE_ENTRY each: KD model width, KO attention output width of a rank, KF FFN width of a rank, head
// dimension, query heads per kv head. Included by the tables of fb_api.cu (one GPU) and fb_decode_tp.cu (ranks), which have to agree in order.
FB_DECODE_ENTRY(512, 512, 1408, 64, 4),       // tiny test decoder
FB_DECODE_ENTRY(512, 512, 1536, 64, 4),       // tiny decoder whose FFN splits into whole groups over 2 ranks
FB_DECODE_ENTRY(512, 256, 768, 64, 4),        // ... and its 2-rank slice
FB_DECODE_ENTRY(640, 640, 1024, 80, 4),       // small decoder with heads of 80 ...
FB_DECODE_ENTRY(640, 384, 512, 80, 4),        // ... whose 2-rank slice reads a widened O window (320 columns in 3 groups)
FB_DECODE_ENTRY(2560, 2560, 8192, 80, 4),     // 3B-class (32 q / 8 kv heads of 80)
#ifndef FB_KERNELS_MINIMAL                    // (a build for kernel experiments keeps only the shapes above)
FB_DECODE_ENTRY(2560, 2560, 8192, 64, 5),     // the reference's native Granite shape (40 q / 8 kv heads of 64)
FB_DECODE_ENTRY(4096, 4096, 14336, 128, 4),   // 8B-class
FB_DECODE_ENTRY(2560, 1280, 4096, 80, 4),     // 3B-class over 2 GPUs
FB_DECODE_ENTRY(2560, 640, 2048, 80, 4),      // 3B-class over 4 GPUs
FB_DECODE_ENTRY(2560, 384, 1024, 80, 4),      // 3B-class over 8 GPUs (320 attention columns inside 3 whole groups)
FB_DECODE_ENTRY(4096, 2048, 7168, 128, 4),    // 8B-class over 2 GPUs
FB_DECODE_ENTRY(4096, 1024, 3584, 128, 4),    // 8B-class over 4 GPUs
FB_DECODE_ENTRY(4096, 512, 1792, 128, 4),     // 8B-class over 8 GPUs
FB_DECODE_ENTRY(2048, 2048, 8192, 64, 4),     // 1B-class (32 q / 8 kv heads of 64)
#endif
#ifdef FB_EXTRA_DECODE_ENTRIES                // further shapes named at build time (build.py: FLINT_B200_EXTRA_SHAPES)
FB_EXTRA_DECODE_ENTRIES
#endif
