// tg_tuning.h -- tile parameters of the kernels: the defaults below, unless the
// sweep in tetragpu_gb300/tune.py found a setting that leads them by more than
// two sweeps differ (python -m tetragpu_gb300.tune --apply writes it into the
// block; tetragpu_gb300/tuning.json keeps the measurements).  A -D on
// the compiler's command line takes precedence (the sweep builds its
// candidates that way).
#pragma once
// BEGIN TUNED
// END TUNED

// defaults of the rest
#ifndef TG_STAR_WIN
#define TG_STAR_WIN 256   // edges a star-pass warp keeps in shared memory
#endif
#ifndef TG_STAR_THREADS
#define TG_STAR_THREADS 128   // threads per star-pass block
#endif
#ifndef TG_STAR_PER
#define TG_STAR_PER 18   // most vertices per warp of the star pass: 126 edges where a vertex owns
                         // seven (a grid; 7.7 on a Delaunay mesh), four full rounds of lanes
                         // (664 us at 128^3 cubes; 694 with 16, 727 with 14; 24 and more go out
                         // early, 696)
#endif
#ifndef TG_STAR_MINB
#define TG_STAR_MINB 10   // resident blocks per SM asked of the star pass
#endif
#ifndef TG_VTS_THREADS
#define TG_VTS_THREADS 128   // threads per VT-sort block
#endif
#ifndef TG_EDGE_ITEMS
#define TG_EDGE_ITEMS 4   // edges per thread of the edge-offset pass
#endif
#ifndef TG_ADJ_WIN
#define TG_ADJ_WIN 256   // VV entries per window of the link adjacency
#endif
#ifndef TG_ADJ_THREADS
#define TG_ADJ_THREADS 128   // threads per link-adjacency block
#endif
