#include <barrier>
#include <atomic>
#include <thread>
#include <vector>
#include <cstdio>
#include <cstdlib>
#include <climits>
#include <random>
#include <numeric>
#include <algorithm>
#include <cstdint>
using std::min; using std::max;
typedef int32_t i32; typedef long i64; typedef uint64_t u64; typedef uint32_t u32;
#define __device__
#define __forceinline__ inline
#define __ldg(p) (*(p))
#define __ffsll __builtin_ffsll
#define PH_ERR_ITER_LIMIT 9
constexpr int MST_SLOTS=8; constexpr u64 NO_OFFER=~0ull;
void set_status(int*s,int v){*s=v;}
void atomicMin(unsigned long long*p,unsigned long long v){std::atomic_ref<unsigned long long> m(*p);auto o=m.load();while(v<o&&!m.compare_exchange_weak(o,v));}
const int T_=13;
std::barrier<> bb(T_); int offered=-1;
struct Bar{ void sync(){bb.arrive_and_wait();} bool any(bool b,int tick){ if(b) *(volatile int*)&offered=tick; bb.arrive_and_wait(); return *(volatile int*)&offered==tick; } };
// pointer jumping of K vertices in lockstep (their loads overlap), each left
// pointing at its root; slots < 0 are padding. A thread writes only its own
// vertices' parents, so no slower walk can put an older ancestor back.
template <int K>
__device__ __forceinline__ void flatten(volatile i32* par, const i32 (&v)[K], bool* bad) {
  i32 p[K];
#pragma unroll
  for (int k = 0; k < K; ++k) p[k] = v[k] >= 0 ? par[v[k]] : -1;
  for (int it = 0; it < (1 << 20); ++it) {
    bool moved = false;
    i32 gp[K];
#pragma unroll
    for (int k = 0; k < K; ++k) gp[k] = p[k] >= 0 ? par[p[k]] : -1;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (gp[k] != p[k]) {
        p[k] = gp[k];
        par[v[k]] = gp[k];
        moved = true;
      }
    if (!moved) return;
  }
  *bad = true;
}

struct MstArgs {
  const i32 *ei, *ej;  // endpoints less vbase are vertices 0 .. n-1
  i64 E, n;
  i32 vbase;
  i32* minv;
  uint8_t* mst;
  i32* comp;
  i64* ncomp;
  int* status;
  int max_rounds;
};

// thread t of T
template <typename Bar>
__device__ void forest(Bar bar, i64 t, i64 T, const MstArgs& a, volatile i32* par, u64* offer) {
  volatile u64* voff = offer;
  const i64 n = a.n, E = a.E;
  for (i64 v = t; v < n; v += T) {
    par[v] = (i32)v;
    offer[v] = NO_OFFER;
    offer[n + v] = NO_OFFER;
    a.minv[v] = INT_MAX;
  }
  {  // the mask: bytes up to a 16-byte boundary, 16-byte stores, bytes
    const i64 head = min(E, (i64)((16 - ((uintptr_t)a.mst & 15)) & 15)), quads = (E - head) / 16;
    uint4* body = reinterpret_cast<uint4*>(a.mst + head);
    for (i64 q = t; q < quads; q += T) body[q] = make_uint4(0, 0, 0, 0);
    for (i64 e = t; e < head; e += T) a.mst[e] = 0;
    for (i64 e = head + 16 * quads + t; e < E; e += T) a.mst[e] = 0;
  }
  if (t == 0) {
    bar.ctl->offered = -1;
    bar.ctl->hooked = 0;
  }
  bool bad = false;
  i32 nu[MST_SLOTS], nv[MST_SLOTS];  // the next pass's edges
  auto load = [&](i64 lo, i64 hi) {
#pragma unroll
    for (int k = 0; k < MST_SLOTS; ++k) {
      const i64 e = lo + t + k * T;
      nu[k] = e < hi ? __ldg(a.ei + e) - a.vbase : -1;
      nv[k] = e < hi ? __ldg(a.ej + e) - a.vbase : -1;
    }
  };
  const i64 full = T * MST_SLOTS;
  i64 lo = 0, hi = min(E, min(full, max(4 * n, T)));
  load(lo, hi);
  bar.sync();
  bool one = n == 1;  // a single component: no later edge can join two
  for (int tick = 0; lo < E && !one;) {
    i32 u[MST_SLOTS], v[MST_SLOTS];
    u32 live = 0;
#pragma unroll
    for (int k = 0; k < MST_SLOTS; ++k) {
      u[k] = nu[k];
      v[k] = nv[k];
      live |= (u[k] >= 0 ? 1u : 0u) << k;
    }
    const i64 base = lo;
    lo = hi;
    hi = min(E, lo + full);
    load(lo, hi);
    for (int round = 0;; ++round, ++tick) {
      if (round >= a.max_rounds) {  // the same for all threads
        if (t == 0) set_status(a.status, PH_ERR_ITER_LIMIT);
        return;
      }
      // offers: the lowest-ranked edge leaving each root; parents of the
      // vertices held are flat (all at a pass's start, roots after a round)
      u64* cur = offer + (size_t)(tick & 1) * n;
      volatile u64* vcur = voff + (size_t)(tick & 1) * n;
      if (base || round) {
#pragma unroll
        for (int k = 0; k < MST_SLOTS; ++k)
          if ((live >> k) & 1u) {
            u[k] = par[u[k]];
            v[k] = par[v[k]];
          }
      }
#pragma unroll
      for (int k = 0; k < MST_SLOTS; ++k)
        if (u[k] == v[k]) live &= ~(1u << k);  // inside one component for good
#pragma unroll
      for (int k0 = 0; k0 < MST_SLOTS; k0 += 4) {
        // a read first: most offers to a busy root lose to a smaller one
        u64 ou[4], ov[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if ((live >> (k0 + k)) & 1u) {
            ou[k] = vcur[u[k0 + k]];
            ov[k] = vcur[v[k0 + k]];
          }
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if ((live >> (k0 + k)) & 1u) {
            const u64 e = (u64)(base + t + (k0 + k) * T) << 32;
            const u64 wu = e | (u32)v[k0 + k], wv = e | (u32)u[k0 + k];
            if (wu < ou[k]) atomicMin((unsigned long long*)&cur[u[k0 + k]], (unsigned long long)wu);
            if (wv < ov[k]) atomicMin((unsigned long long*)&cur[v[k0 + k]], (unsigned long long)wv);
          }
      }
      if (!bar.any(live != 0, tick)) {
        if (round) {  // every vertex to its root: the next pass's edges are met with one load
          for (i64 x0 = t; x0 < n; x0 += 4 * T) {
            i32 x[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) x[k] = x0 + k * T < n ? (i32)(x0 + k * T) : -1;
            flatten(par, x, &bad);
          }
          bar.sync();
        }
        tick += 2;  // the array of this round is the clean one, and any() takes each tick once
        break;
      }
      // hooks; the other offer array (last read in the previous round) is cleared
      u64* idle = offer + (size_t)((tick + 1) & 1) * n;
      u64 hooked = 0;  // of the thread's first 64 vertices
      int hooks = 0;
      i64 j = 0;
      for (i64 x = t; x < n; x += T, ++j) {
        if (par[x] != (i32)x) continue;
        idle[x] = NO_OFFER;
        const u64 w = vcur[x];
        if (w == NO_OFFER) continue;
        const i32 e = (i32)(w >> 32), o = (i32)(w & 0xffffffffull);
        a.mst[e] = 1;
        if ((vcur[o] >> 32) == (u64)e && o > (i32)x) continue;  // mutual choice: the larger root hooks
        par[x] = o;
        ++hooks;
        hooked |= j < 64 ? 1ull << j : 0ull;
      }
      hooks = __reduce_add_sync(0xffffffffu, hooks);
      if ((threadIdx.x & 31) == 0 && hooks) atomicAdd(&bar.ctl->hooked, hooks);
      bar.sync();
      one = *(volatile int*)&bar.ctl->hooked == n - 1;  // the same for all: next added to after a barrier
      if (one) break;
      if (j <= 64) {
        while (hooked) {
          i32 x[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            x[k] = hooked ? (i32)(t + (i64)(__ffsll((long long)hooked) - 1) * T) : -1;
            hooked &= hooked - 1;
          }
          flatten(par, x, &bad);
        }
      } else {  // more vertices a thread than the mask holds: all of them
        for (i64 x0 = t; x0 < n; x0 += 4 * T) {
          i32 x[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) x[k] = x0 + k * T < n ? (i32)(x0 + k * T) : -1;
          flatten(par, x, &bad);
        }
      }
      bar.sync();
    }
  }
  if (one) {
    for (i64 x = t; x < n; x += T) a.comp[x] = a.vbase;
    if (t == 0) atomicAdd((unsigned long long*)a.ncomp, 1ull);
    if (bad) set_status(a.status, PH_ERR_ITER_LIMIT);
    return;
  }
  // labels: the smallest vertex of each component, and the component count.
  // Vertices ascend over the lanes, so the first lane of those with one root
  // holds the least of them.
  for(i64 x=t;x<n;x+=T){ i32 r=par[x]; if(par[r]!=r) {printf("notflat\n");abort();} std::atomic_ref<i32> m(a.minv[r]); i32 o=m.load(); while(x<o&&!m.compare_exchange_weak(o,(i32)x)); if(r==x) std::atomic_ref<i64>(*a.ncomp)++; }
  bar.sync();
  for (i64 x = t; x < n; x += T) a.comp[x] = a.vbase + *(volatile i32*)(a.minv + par[x]);
  if (bad) set_status(a.status, PH_ERR_ITER_LIMIT);
}


int main(){ std::mt19937 g(1); for(int it=0;it<400;++it){ i64 n=1+g()%(it%3?300:3000), E=g()%(it%5?4000:20000); std::vector<i32> ei(E),ej(E); for(i64 e=0;e<E;++e){ei[e]=g()%n;ej[e]=g()%n;} if(it%4==0){std::vector<i32> p(n);std::iota(p.begin(),p.end(),0);for(i64 k=0;k<min(E,n);++k){ei[k]=k;ej[k]=(k+1)%n;} for(i64 k=E-1;k>0;--k){i64 j=g()%(k+1);std::swap(ei[k],ei[j]);std::swap(ej[k],ej[j]);}}
 std::vector<i32> par(n),minv(n),comp(n); std::vector<u64> off(2*n); std::vector<uint8_t> mst(E+1); i64 nc=77; int st=0; offered=-1;
 int mr=2; while((i64(1)<<(mr-2))<n&&mr<64)++mr; mr+=4;
 MstArgs a{ei.data(),ej.data(),E,n,minv.data(),mst.data(),comp.data(),&nc,&st,mr};
 std::vector<std::thread> th; for(int t=0;t<T_;++t) th.emplace_back([&,t]{ forest(Bar{},t,T_,a,par.data(),off.data()); }); for(auto&x:th)x.join();
 std::vector<i32> q(n);std::iota(q.begin(),q.end(),0); auto f=[&](i32 v){while(q[v]!=v)v=q[v]=q[q[v]];return v;}; i64 c=n; for(i64 e=0;e<E;++e){i32 x=f(ei[e]),y=f(ej[e]); int w=x!=y; if(w){q[max(x,y)]=min(x,y);--c;} if(w!=mst[e]){printf("bad mask it %d n %ld E %ld e %ld st %d\n",it,n,E,e,st);return 1;}}
 for(i64 v=0;v<n;++v) if(comp[v]!=f(v)){printf("bad comp\n");return 1;} if(nc!=c||st){printf("bad nc\n");return 1;} }
 puts("ok"); }
