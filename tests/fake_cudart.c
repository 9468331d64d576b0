/* Host stand-ins for the CUDA runtime calls of libsesgb.so, for tests without a GPU (LD_PRELOAD): device memory is host
 * memory, kernels do not run, launches are counted, and allocations can be made to fail. A counter record copied to the host
 * can be given a value, as a kernel would have left it. */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

static int          fail_mallocs, last_error;
static unsigned     launches, mallocs, frees, poke_word, poke_value, poke_left;
static const void * fill_from;
static unsigned long long bytes;
static size_t       fill_bytes;

void     fake_fail( int n ) { fail_mallocs = n; }
unsigned fake_launches( void ) { return launches; }
unsigned long long fake_bytes( void ) { return bytes; } /* allocated so far */
unsigned fake_live( void ) { return mallocs - frees; }
/* the next `times` copies of a counter record (100 to 255 bytes) to the host have `value` in word `word` */
void fake_poke( unsigned word, unsigned value, unsigned times )
{
    poke_word  = word;
    poke_value = value;
    poke_left  = times;
}

/* copies of exactly n bytes to the host read from p */
void fake_fill( const void * p, unsigned n )
{
    fill_from  = p;
    fill_bytes = n;
}

int cudaMalloc( void ** p, size_t n )
{
    if ( fail_mallocs > 0 )
    {
        fail_mallocs--;
        return last_error = 2; /* out of memory */
    }
    mallocs++;
    bytes += n;
    *p = calloc( n ? n : 1, 1 );
    return 0;
}
int cudaFree( void * p )
{
    frees += p != NULL;
    free( p );
    return 0;
}
int cudaHostAlloc( void ** p, size_t n, unsigned flags )
{
    (void)flags;
    *p = calloc( n, 1 );
    return 0;
}
int cudaMallocHost( void ** p, size_t n ) { return cudaHostAlloc( p, n, 0 ); }
int cudaFreeHost( void * p )
{
    free( p );
    return 0;
}
int cudaMemcpy( void * d, const void * s, size_t n, int kind )
{
    memcpy( d, kind == 2 && fill_from && n == fill_bytes ? fill_from : s, n );
    if ( kind == 2 && n >= 100 && n < 256 && poke_left )
    {
        poke_left--;
        ( (uint32_t *)d )[ poke_word ] = poke_value;
    }
    return 0;
}
int cudaMemcpyAsync( void * d, const void * s, size_t n, int kind, void * stream )
{
    (void)stream;
    return cudaMemcpy( d, s, n, kind );
}
int cudaMemset( void * d, int v, size_t n )
{
    memset( d, v, n );
    return 0;
}
int cudaMemsetAsync( void * d, int v, size_t n, void * stream )
{
    (void)stream;
    return cudaMemset( d, v, n );
}
int cudaGetLastError( void )
{
    const int e = last_error;
    last_error  = 0;
    return e;
}
const char * cudaGetErrorString( int e ) { return e ? "out of memory" : "no error"; }

static int launched( void )
{
    launches++;
    return 0;
}
int __cudaLaunchKernel( void ) { return launched(); }
int cudaLaunchKernel( void ) { return launched(); }
int cudaLaunchKernelExC( void ) { return launched(); }
int cudaGraphLaunch( void ) { return launched(); }
int __cudaGetKernel( void ** k, const void * f )
{
    *k = (void *)f;
    return 0;
}
int cudaDeviceGetAttribute( int * v )
{
    *v = 152;
    return 0;
}
int cudaGetDevice( int * d )
{
    *d = 0;
    return 0;
}
int cudaSetDevice( void ) { return 0; }
int cudaDeviceSynchronize( void ) { return 0; }
int cudaStreamSynchronize( void ) { return 0; }
int cudaFuncSetAttribute( void ) { return 0; }
int cudaStreamBeginCapture( void ) { return 0; }
int cudaStreamWaitEvent( void ) { return 0; }
int cudaEventRecord( void ) { return 0; }
int cudaEventRecordWithFlags( void ) { return 0; }

static int made( void ** p )
{
    static int handle;
    *p = &handle;
    return 0;
}
int cudaStreamCreateWithFlags( void ** p ) { return made( p ); }
int cudaEventCreate( void ** p ) { return made( p ); }
int cudaEventCreateWithFlags( void ** p ) { return made( p ); }
int cudaStreamEndCapture( void * stream, void ** g ) { return made( g ); }
int cudaGraphInstantiate( void ** g ) { return made( g ); }
int cudaStreamDestroy( void ) { return 0; }
int cudaEventDestroy( void ) { return 0; }
int cudaGraphDestroy( void ) { return 0; }
int cudaGraphExecDestroy( void ) { return 0; }
